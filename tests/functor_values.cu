// A vertex-centric functor over a value of VALUE_WORDS four-byte words, ints and
// floats in turn, each summed (ONE_WORD: the last one only): every expand of the
// engine has to build for it and give the same sums.
#include "engine/executor.cuh"
using namespace gsw;
using G = device_graph_t<CSR, Empty>;

struct value_t {
  int a[(VALUE_WORDS + 1) / 2];
#if VALUE_WORDS > 1
  float b[VALUE_WORDS / 2];
#endif
};

struct sender_t {
  int active;
  value_t sends;
};

struct Gather : Functor<VC, value_t, sender_t, Empty> {
  __device__ Status filter(int v, G) { return ra_of(v)->active ? Active : Inactive; }
  __device__ value_t emit(int v, Empty *, G) { return ra_of(v)->sends; }
  __device__ bool cond(int, value_t, G) { return true; }
#ifdef ONE_WORD
  __device__ bool comp(value_t *v, value_t m, G) {
    v->b[VALUE_WORDS / 2 - 1] += m.b[VALUE_WORDS / 2 - 1];
    return true;
  }
  __device__ bool compAtomic(value_t *v, value_t m, G) {
    atomicAdd(&v->b[VALUE_WORDS / 2 - 1], m.b[VALUE_WORDS / 2 - 1]);
    return true;
  }
#else
  __device__ bool comp(value_t *v, value_t m, G) {
    for (int i = 0; i < (VALUE_WORDS + 1) / 2; ++i) v->a[i] += m.a[i];
#if VALUE_WORDS > 1
    for (int i = 0; i < VALUE_WORDS / 2; ++i) v->b[i] += m.b[i];
#endif
    return true;
  }
  __device__ bool compAtomic(value_t *v, value_t m, G) {
    for (int i = 0; i < (VALUE_WORDS + 1) / 2; ++i) atomicAdd(&v->a[i], m.a[i]);
#if VALUE_WORDS > 1
    for (int i = 0; i < VALUE_WORDS / 2; ++i) atomicAdd(&v->b[i], m.b[i]);
#endif
    return true;
  }
#endif
};

// One level under one variant: the active vertices send their values to the others
// (all: every vertex to every vertex).  Host arrays; sums are n rows of VALUE_WORDS
// words, added to in place.  passes: levels run in a row.
extern "C" int gather_level(int n, long long m, const int64_t *off, const int *col, const int64_t *roff,
                            const int *rcol, int directed, const sender_t *senders, value_t *sums, int dir, int fmt,
                            int lb, int all, int pruning, int passes) {
  auto dev = [](const void *h, size_t bytes) {
    void *d = nullptr;
    if (cudaMalloc(&d, bytes + 16) == cudaSuccess) cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice);
    return d;
  };
  std::vector<int> deg(n), rdeg(n);
  for (int v = 0; v < n; ++v) deg[v] = (int)(off[v + 1] - off[v]), rdeg[v] = (int)(roff[v + 1] - roff[v]);
  G g;
  g.dg_row_off = (int64_t *)dev(off, 8 * ((size_t)n + 1));
  g.dgr_row_off = (int64_t *)dev(roff, 8 * ((size_t)n + 1));
  g.dg_adj_list = (int *)dev(col, 4 * (size_t)m);
  g.dgr_adj_list = (int *)dev(rcol, 4 * (size_t)m);
  g.dg_odegree = (int *)dev(deg.data(), 4 * (size_t)n);
  g.dgr_odegree = (int *)dev(rdeg.data(), 4 * (size_t)n);
  g.dg_edgedata = g.dgr_edgedata = nullptr;
  g.nvertexs = n;
  g.nedges = m;
  g.level = 0;
  g.directed = directed != 0;
  Gather f;
  memset(&f.data.zero, 0, sizeof(value_t));
  f.data.size = n;
  f.data.dg_wa = (value_t *)dev(sums, sizeof(value_t) * (size_t)n);
  f.data.dg_ra = (sender_t *)dev(senders, sizeof(sender_t) * (size_t)n);
  stat_t stats;
  feature_t fets;
  config_t conf;
  inspector_t inspector;
  selector_t selector;
  executor_t executor;
  executor.insp = &inspector;
  fets.centric = VC;
  fets.pattern = ASSO;
  fets.fromall = fets.toall = all != 0;
  fets.nvertexs = n;
  fets.nedges = m;
  fets.avg_deg = (double)m / n;
  fets.use_root = -1;
  conf.conf_pruning = pruning != 0;
  conf.force.has_direction = conf.force.has_asfmt = conf.force.has_lb = conf.force.has_fusion = true;
  conf.force.d = dir ? Pull : Push;
  conf.force.asf = fmt ? Bitmap : Queue;
  conf.force.lb = (LB)lb;
  conf.force.fusion = Standalone;
  init_conf_impl(stats, fets, conf, g, f, 0.0, fets.avg_deg, false);
  conf.conf_first_round = false;  // inspect
  active_set_t as = build_active_set(n, conf.conf_qmode);
  as.init(ALL_INACTIVE);
  for (int i = 0; i < passes && ok(); ++i) {
    inspector.inspect(as, g, f, stats, fets, conf);
    selector.select(stats, fets, conf);
    executor.filter(as, g, f, stats, fets, conf);
    executor.expand(as, g, f, stats, fets, conf);
  }
  cudaStreamSynchronize(stream());
  const cudaError_t e = cudaMemcpy(sums, f.data.dg_wa, sizeof(value_t) * (size_t)n, cudaMemcpyDeviceToHost);
  const int code = ok() ? (int)e : 1000 + (int)err().code;
  executor.destroy();
  as.destroy();
  stats.destroy();
  for (const void *p : {(const void *)g.dg_row_off, (const void *)g.dgr_row_off, (const void *)g.dg_adj_list,
                        (const void *)g.dgr_adj_list, (const void *)g.dg_odegree, (const void *)g.dgr_odegree,
                        (const void *)f.data.dg_wa, (const void *)f.data.dg_ra})
    cudaFree((void *)p);
  return code;
}
