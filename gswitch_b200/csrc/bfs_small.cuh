// BFS of a small graph in one launch.
//
// The level loop spends about 30 us a level on a graph that fits a few SMs: an
// inspection (10 us whatever the size), a queue build of three launches, an
// expand and a round trip to the host, to move a few thousand arcs.  A small
// graph's BFS therefore runs whole in one cooperative launch, from the initial
// levels to the traversed-edge count, with one grid barrier a level.
// A discovered vertex is appended as pieces of at most SB_PIECE arcs, so a level
// is balanced without a scan of its degrees: a warp takes a piece at a time.
// What bounds it is the chain of a level: piece, columns, levels of their
// vertices, the append and the barrier, about 5 us.  Every level pushes; on
// larger graphs the pull's early exit saves more than the loop costs.  SB_MAX_*:
// one call, this against the loop (timed, its events included), is 73 against 292
// us on RMAT 2^10, 144 against 384 on 2^16, 198 against 386 on 2^17 (3.7 M arcs),
// 271 against 412 on 2^18 with 3.9 M arcs, 269 against 360 on G(2^18, 2^21), 177
// against 235 on a star of 2^18.  Past the line the gain runs out: RMAT 2^18 with
// 7.6 M arcs 294 against 400, 2^19 with 15.5 M 467 against 487, 2^20 with 31 M 770
// against 656, G(2^20, 2^21) 949 against 766.  Long graphs keep a level below the
// loop's persistent one: a lattice of 512 x 512 with 633 levels 3.5 against 5.6 ms,
// of 64 x 4,096 with 3,902 levels 18.8 against 31.8 ms, a chain of 12,527 levels 43
// against 84 ms.
#pragma once
#include "engine/executor.cuh"

namespace gsw {

constexpr int SB_THREADS = 1024;
constexpr int SB_PIECE = 128;  // arcs a warp takes at a time, four to a lane in flight
constexpr int64_t SB_MAX_VERTICES = 1 << 18;
constexpr int64_t SB_MAX_ARCS = 1 << 22;

struct sb_piece_t {
  int beg, len;  // columns [beg, beg + len)
};
struct sb_state_t {
  unsigned bar[3];              // grid barrier: arrivals, generation, error word
  int size[3];                  // pieces of a level, by level modulo 3
  unsigned long long reached;   // degree sum of the reached vertices
  int levels;                   // levels expanded
  int status;                   // 0 done, 2 barrier timeout
};

// appends v's arcs in pieces; every lane of the warp calls it
__device__ __forceinline__ void sb_append(const int64_t *off, bool found, int v, sb_piece_t *q, int *size,
                                          unsigned long long &reached) {
  if (!__any_sync(FULL, found)) return;
  int beg = 0, deg = 0;
  if (found) {
    const int64_t b = __ldg(off + v);
    beg = (int)b;
    deg = (int)(__ldg(off + v + 1) - b);
    reached += deg;
  }
  const int np = (deg + SB_PIECE - 1) / SB_PIECE;
  const int incl = warp_inclusive_sum(np);
  const int total = __shfl_sync(FULL, incl, 31);
  if (total == 0) return;
  int base = 0;
  if (lane_id() == 0) base = atomicAdd(size, total);
  base = __shfl_sync(FULL, base, 0);
  sb_piece_t *out = q + base + incl - np;
  if (np <= 2)
    for (int k = 0; k < np; ++k) out[k] = sb_piece_t{beg + k * SB_PIECE, MIN(SB_PIECE, deg - k * SB_PIECE)};
  // long rows: the whole warp writes one's pieces
  for (unsigned m = __ballot_sync(FULL, np > 2); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int n1 = __shfl_sync(FULL, np, src), b1 = __shfl_sync(FULL, beg, src), d1 = __shfl_sync(FULL, deg, src);
    sb_piece_t *o1 = q + base + __shfl_sync(FULL, incl, src) - n1;
    for (int k = lane_id(); k < n1; k += 32) o1[k] = sb_piece_t{b1 + k * SB_PIECE, MIN(SB_PIECE, d1 - k * SB_PIECE)};
  }
}

// q0, q1: room for n + arcs / SB_PIECE pieces each (a vertex is found once)
__global__ void __launch_bounds__(SB_THREADS, 1)
    k_bfs_small(device_graph_t<CSR, Empty> g, int root, const int *roots, int nroots, int *level, sb_piece_t *q0,
                sb_piece_t *q1, sb_state_t *S, unsigned long long budget_ns) {
  sb_piece_t *const q[2] = {q0, q1};
  const int lane = lane_id();
  const int n = g.nvertexs;
  const int nwarps = gridDim.x * (SB_THREADS / 32), gw = blockIdx.x * (SB_THREADS / 32) + warp_id();
  unsigned gen = 0;
  auto barrier = [&] { return grid_barrier(S->bar, S->bar + 1, S->bar + 2, gen, budget_ns); };
  unsigned long long reached = 0;
  for (int v = blockIdx.x * SB_THREADS + threadIdx.x; v < n; v += gridDim.x * SB_THREADS)
    level[v] = roots == nullptr && v == root ? 0 : -1;
  if (roots == nullptr && gw == 0) sb_append(g.dg_row_off, lane == 0, root, q[0], &S->size[0], reached);
  bool okk = barrier();
  if (roots && okk) {  // a root listed twice is one root
    for (int i = gw * 32; i < nroots; i += nwarps * 32) {
      const int v = i + lane < nroots ? roots[i + lane] : -1;
      sb_append(g.dg_row_off, v >= 0 && atomicCAS(level + v, -1, 0) == -1, v, q[0], &S->size[0], reached);
    }
    okk = barrier();
  }
  int L = 0;
  while (okk) {
    const int np = ((volatile int *)S->size)[L % 3];
    if (np == 0) break;
    if (blockIdx.x == 0 && threadIdx.x == 0) S->size[(L + 2) % 3] = 0;  // last read before the previous barrier
    for (int p = gw; p < np; p += nwarps) {
      const sb_piece_t pc = q[L & 1][p];
      int u[SB_PIECE / 32];
      bool found[SB_PIECE / 32];
#pragma unroll
      for (int k = 0; k < SB_PIECE / 32; ++k)
        u[k] = 32 * k + lane < pc.len ? __ldg(g.dg_adj_list + pc.beg + 32 * k + lane) : -1;
      // a level may be older than the current one: the compare-and-swap decides
#pragma unroll
      for (int k = 0; k < SB_PIECE / 32; ++k) found[k] = u[k] >= 0 && level[u[k]] < 0;
#pragma unroll
      for (int k = 0; k < SB_PIECE / 32; ++k) found[k] = found[k] && atomicCAS(level + u[k], -1, L + 1) == -1;
#pragma unroll
      for (int k = 0; k < SB_PIECE / 32; ++k)
        sb_append(g.dg_row_off, found[k], u[k], q[(L + 1) & 1], &S->size[(L + 1) % 3], reached);
    }
    okk = barrier();
    ++L;
  }
  reached = warp_sum(reached);
  if (lane == 0 && reached) atomicAdd(&S->reached, reached);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S->levels = L;
    S->status = okk ? 0 : 2;
  }
}

}  // namespace gsw
