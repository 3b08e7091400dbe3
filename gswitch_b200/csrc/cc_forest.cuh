// Connected components by sampled hooking (Afforest: Sutton, Ben-Nun, Barak,
// IPDPS 2018).
//
// The edge-centric loop (application/cc.cu:82-108) reads the whole edge list at
// least twice, once to hook and once to find that every edge is settled, with
// two or more random label reads per edge: 1.18 ms for the 64 M edges of RMAT
// 2^22, and the list has to be built first.  Most of those edges join vertices
// that a few edges per vertex have already joined.  Here every vertex first
// hooks along three of its arcs, the most common label is read off a sample,
// and only the vertices outside that component go through all of their arcs.
// An arc with one end outside is seen from that end, so none is missed
// (provided that each arc is listed from both ends, which k_arc_pairs checks).
// Hooking always puts the larger root under the smaller one, so a component's
// label is its smallest vertex, as in the loop.
// The trees are flattened before every pass that climbs them: ids that follow a
// path or a mesh make the first trees as deep as the graph is long, and hooking
// climbs one vertex at a time (two interleaved paths of 2^20 vertices: 0.08 ms,
// 89 ms with one flatten before the last pass).
// What bounds it: ten short passes over the vertices, each with a random label
// read per vertex: 158 us on RMAT 2^22, where the loop's two inspections, two
// hooking passes and pointer jumps took 1,183 us.
#pragma once
#include "engine/executor.cuh"
#include "graphgen.cuh"

namespace gsw {

constexpr int CC_THREADS = 256;
constexpr int CC_ROW_WARP = 16;     // arcs from which a warp takes a row together
constexpr int CC_ROW_PIECE = 4096;  // and from which it is cut for several warps
constexpr int CC_SAMPLE = 1024;

struct cc_state_t {
  int common;  // the most common label
  int pieces;  // listed row pieces
};
struct row_facts_t {
  unsigned long long up;       // arcs v -> u with u > v (the undirected edges)
  unsigned long long balance;  // sum over arcs of +-hash(smaller, larger): 0 when each is listed from both ends
  long long descents;          // inside rows (k_row_descents): 0 when every row ascends
};
struct cc_piece_t {
  int64_t beg;
  int v, len;
};

// The passes are short, so each is set up while the one before still runs
// (programmatic dependent launch: the next may be launched at once, and waits here
// for everything the one before writes).  With ten passes a call on RMAT 2^16 takes
// 50 us, 69 us with plain launches (61 us with eight); 2^22 179 and 194 us.
__device__ __forceinline__ void cc_begin() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}
template <typename... P, typename... A>
inline void cc_launch(void (*kern)(P...), int grid, int threads, bool first, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream();
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = first ? 0 : 1;  // whatever ran before the first pass ends before it
  if (!GSW_CUDA(cudaLaunchKernelEx(&cfg, kern, P(args)...))) GSW_LAUNCHED();
}

// Joins the trees of u and v: the larger root goes under the smaller.  Labels
// are read through the L1: an old label is still an ancestor (labels only move
// towards the root), and the root that all of a large component reads would
// otherwise be one L2 address for the whole grid (two link passes and a flatten
// took 500 us on RMAT 2^22 with uncached reads).  The compare-and-swap decides on the current label and
// returns it, so every step leaves max(a, b) smaller.
__device__ __forceinline__ void cc_link(int *comp, int u, int v) {
  int a = comp[u], b = comp[v];
  while (a != b) {
    const int hi = max(a, b), lo = min(a, b);
    int p = comp[hi];
    if (p == hi) p = atomicCAS(comp + hi, hi, lo);
    if (p == hi || p == lo) return;
    a = p;
    b = lo;
  }
}

// every vertex under its first neighbour where that is the smaller: a forest,
// since parents only get smaller
__global__ void __launch_bounds__(CC_THREADS) k_cc_start(const int64_t *off, const int *col, int64_t n, int *comp) {
  cc_begin();
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = __ldg(off + v), e = __ldg(off + v + 1);
    comp[v] = b < e ? min((int)v, __ldg(col + b)) : (int)v;
  }
}
// along the second arc, or the last
__global__ void __launch_bounds__(CC_THREADS) k_cc_link_one(const int64_t *off, const int *col, int64_t n, int *comp,
                                                            bool last) {
  cc_begin();
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = __ldg(off + v), e = __ldg(off + v + 1);
    if (e - b > (last ? 2 : 1)) cc_link(comp, (int)v, __ldg(col + (last ? e - 1 : b + 1)));
    else if (e - b == 1) cc_link(comp, (int)v, __ldg(col + b));
  }
}
// every vertex under its root (roots stay roots meanwhile).  Each step is
// written at once: threads further down the same chain then jump over what this
// one has climbed, and a chain of n vertices takes log n steps and not n.
__global__ void __launch_bounds__(CC_THREADS) k_cc_flatten(int *comp, int64_t n) {
  cc_begin();
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    int p = comp[v], q;
    while (p != (q = comp[p])) comp[v] = p = q;
  }
}
// the most common label among CC_SAMPLE vertices spread over the ids
__global__ void __launch_bounds__(CC_SAMPLE) k_cc_common(const int *comp, int64_t n, cc_state_t *S) {
  cc_begin();
  constexpr int SLOTS = 4 * CC_SAMPLE;
  __shared__ int s_key[SLOTS], s_cnt[SLOTS];
  __shared__ unsigned long long s_best;
  for (int i = threadIdx.x; i < SLOTS; i += blockDim.x) s_key[i] = -1, s_cnt[i] = 0;
  if (threadIdx.x == 0) s_best = 0;
  __syncthreads();
  const int l = comp[sm64(threadIdx.x) % (uint64_t)n];
  unsigned at = (unsigned)sm64((uint64_t)l) % SLOTS;
  for (;;) {  // at most CC_SAMPLE labels in four times as many slots
    const int k = atomicCAS(&s_key[at], -1, l);
    if (k == -1 || k == l) break;
    at = (at + 1) % SLOTS;
  }
  const int c = atomicAdd(&s_cnt[at], 1) + 1;
  atomicMax(&s_best, ((unsigned long long)c << 32) | (unsigned)l);
  __syncthreads();
  if (threadIdx.x == 0) {
    S->common = (int)(unsigned)s_best;
    S->pieces = 0;
  }
}
// all arcs of the vertices outside the common component; long rows are listed.
// A vertex whose tree is hooked under the common label meanwhile may be passed
// over: it is joined already, and whatever it leaves out is seen from the other
// end.
__global__ void __launch_bounds__(CC_THREADS) k_cc_rest(const int64_t *off, const int *col, int64_t n, int *comp,
                                                        cc_state_t *S, cc_piece_t *piece) {
  cc_begin();
  const int common = S->common, lane = lane_id();
  for (int64_t v0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~int64_t(31); v0 < n;
       v0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = v0 + lane;
    int64_t b = 0;
    int deg = 0;
    if (v < n && comp[v] != common) {
      b = __ldg(off + v);
      deg = (int)(__ldg(off + v + 1) - b);
    }
    if (deg >= CC_ROW_PIECE) {
      const int np = (deg + CC_ROW_PIECE - 1) / CC_ROW_PIECE;
      const int at = atomicAdd(&S->pieces, np);
      for (int k = 0; k < np; ++k)
        piece[at + k] = cc_piece_t{b + (int64_t)k * CC_ROW_PIECE, (int)v, MIN(CC_ROW_PIECE, deg - k * CC_ROW_PIECE)};
      deg = 0;
    }
    for (unsigned m = __ballot_sync(FULL, deg >= CC_ROW_WARP); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int u = (int)v0 + src, d = __shfl_sync(FULL, deg, src);
      const int64_t rb = __shfl_sync(FULL, b, src);
      for (int k = lane; k < d; k += 32) cc_link(comp, u, __ldg(col + rb + k));
    }
    if (deg < CC_ROW_WARP)
      for (int k = 0; k < deg; ++k) cc_link(comp, (int)v, __ldg(col + b + k));
  }
}
__global__ void __launch_bounds__(CC_THREADS) k_cc_pieces(const int *col, int *comp, const cc_state_t *S,
                                                          const cc_piece_t *piece) {
  cc_begin();
  const int np = S->pieces;
  for (int i = blockIdx.x; i < np; i += gridDim.x) {
    const cc_piece_t p = piece[i];
    for (int k = threadIdx.x; k < p.len; k += blockDim.x) cc_link(comp, p.v, __ldg(col + p.beg + k));
  }
}

// Is every arc listed from both ends?  Each pair adds its hash where the row is
// the smaller end and takes it away where it is the larger; a sum of 0 over all
// arcs is the answer (of 2^64 values, by chance, for a graph that is not).
// Also counts the edges.  One warp per 256 slots of the rows, as the all-to-all
// expands lay them out.
__global__ void __launch_bounds__(EXPAND_THREADS) k_arc_pairs(const int64_t *off, const int *col, int64_t n, int64_t m,
                                                              const int *tile_lo, int64_t ntiles, row_facts_t *F) {
  __shared__ unsigned short s_begs[ALL_WARPS][ALL_TILE + 2];
  const int lane = lane_id();
  unsigned short *s_beg = s_begs[warp_id()];
  unsigned long long up = 0, balance = 0;
  for (int64_t t = (int64_t)blockIdx.x * ALL_WARPS + warp_id(); t < ntiles; t += (int64_t)gridDim.x * ALL_WARPS) {
    const int lo = tile_lo[t], hi = t + 1 < ntiles ? tile_lo[t + 1] : (int)n - 1;
    const int64_t ea = t * ALL_TILE - lo, eb = t + 1 < ntiles ? (t + 1) * ALL_TILE - hi : m;
    const int cnt = hi - lo + 1, ne = (int)(eb - ea);
    __syncwarp();
    for (int j = lane; j <= cnt; j += 32) {
      const int64_t b = __ldg(off + lo + j) - ea;
      s_beg[j] = (unsigned short)(b < 0 ? 0 : (b > ne ? ne : b));
    }
    __syncwarp();
    for (int e = lane; e < ne; e += 32) {
      const int v = lo + tile_owner(s_beg, cnt, e), u = ld_stream(col + ea + e);
      if (u > v) {
        ++up;
        balance += sm64(((uint64_t)v << 32) | (unsigned)u);
      } else if (u < v) {
        balance -= sm64(((uint64_t)u << 32) | (unsigned)v);
      }
    }
  }
  up = warp_sum(up);
  balance = warp_sum(balance);
  if (lane == 0) {
    atomicAdd(&F->up, up);
    atomicAdd(&F->balance, balance);
  }
}

}  // namespace gsw
