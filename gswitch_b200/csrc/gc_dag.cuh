// Graph colouring in dependency order.
//
// The colouring functor (application/gc.cu:15-43) gives a vertex the first
// level at which no uncoloured in-neighbour has a larger id.  So a vertex's
// colour is one more than the largest colour among its in-neighbours with
// larger ids, and it is settled when the last of them is.  The level loop
// finds this by sweeping every arc of every uncoloured vertex at every level:
// on RMAT 2^18 (7.6 M arcs, 732 colours) 732 sweeps, 75 ms, nearly all of it
// re-reading arcs whose answer has not changed.  Here each vertex holds the
// number of its uncoloured larger in-neighbours; colouring v takes one from
// every smaller out-neighbour, and one that reaches zero joins the next
// level's frontier.  Every arc is used once, so what bounds it is the chain of
// dependent levels (column, counter, the vertices that reached zero): 4.4 ms in
// all for that graph, 5.9 us a level.
//
// One cooperative launch runs all levels.  A frontier of few vertices and arcs
// stays on one CTA, in shared memory, where a level ends at a CTA barrier; a
// larger one is spread over the grid with a grid barrier per level.  On one CTA
// a scan deals the level's arcs out evenly, GC_ROWS to a thread and all in
// flight (a warp to a vertex took 12.5 us a level, with up to a dozen vertices
// in turn), and the line GC_SMALL_ARCS is one such round.
// A long row of a large level is cut into pieces, taken after one more grid
// barrier: left to the warps of its vertex, a row of 2^20 smaller neighbours in a
// frontier of 6,000 vertices took 27 ms (a lone warp); cut, 0.07 ms.  The barrier
// is spent only where such a row is in the frontier.
// The rows have to be sorted, so that a vertex's smaller neighbours are the
// front of its row; the caller checks (k_row_descents).  An undirected graph
// also has to list each arc from both ends (k_arc_pairs): the counters come from
// a vertex's own row and are taken down along its neighbours' rows.  Any other
// graph keeps the level loop.
#pragma once
#include "engine/executor.cuh"

namespace gsw {

constexpr int GC_THREADS = 1024;
constexpr int GC_SMALL_VERTICES = 1024;  // frontier one CTA takes
constexpr int GC_SMALL_ARCS = 8192;      // and the arcs it sends along: eight rounds of the CTA
constexpr int GC_SMALL_LEVELS = 4096;    // levels before the waiting CTAs see a barrier again
constexpr int GC_ROWS = GC_SMALL_ARCS / GC_THREADS;  // arcs of a thread in a small level
constexpr int GC_LAUNCH_LEVELS = 1 << 16;
constexpr int GC_BATCH = 2;     // arcs of a lane in flight in a large level
constexpr int GC_LONG = 1024;   // in a large level, longer rows (per warp that shares one)
constexpr int GC_PIECE = 256;   // are cut into pieces of so many arcs for the whole grid

// A frontier, as it is handed on: read by every warp of the grid after a barrier,
// so it is one 16-byte load (4,736 warps meet at one L2 address each time: a word
// more, read by itself, took G(2^18, 2^22) from 0.97 to 1.22 ms).
struct alignas(16) gc_front_t {
  unsigned arcs;  // the arcs it sends along (capped: compared with what one CTA takes)
  int size;       // its vertices that have any
  int level;      // its colour
  int longs;      // it may have rows of GC_LONG arcs or more
};
// one that the grid builds
struct alignas(16) gc_next_t {
  unsigned long long arcs;
  int size;
  int longs;
};
struct gc_state_t {
  unsigned bar[3];  // grid barrier: arrivals, generation, error word
  int pieces[3];    // what a level's long rows were cut into
  // frontiers the grid builds, by the number of grid-wide levels modulo 3: a
  // slot is cleared two levels after it was read, so a barrier lies between (so are
  // the pieces' counts)
  gc_next_t next[3];
  // what CTA 0 hands back when it leaves its own levels, by the parity of such
  // hand-overs: a slot is written again only after every CTA passed the next one
  gc_front_t pub[2];
  gc_front_t at;                  // where the launch stopped
  unsigned long long coloured;    // vertices that have their colour
  int status;                     // 0 done, 1 launch's level cap, 2 barrier timeout
};
struct gc_piece_t {
  int64_t beg;  // columns [beg, beg + len)
  int len;
};
// room for the pieces of a level: a row is listed once
inline int64_t gc_pieces(int64_t arcs) { return arcs / GC_PIECE + arcs / GC_LONG + 1; }

// Descents col[e] > col[e+1] along the whole column array, minus those where a
// row starts: 0 when every row is sorted.
__global__ void k_row_descents(const int64_t *off, const int *col, int64_t n, int64_t m, long long *out) {
  long long d = 0;
  const int64_t T = (int64_t)gridDim.x * blockDim.x, t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t e = t0; e + 1 < m; e += T) d += __ldg(col + e) > __ldg(col + e + 1);
  for (int64_t v = t0; v < n; v += T) {
    const int64_t b = __ldg(off + v);
    if (b > 0 && b < __ldg(off + v + 1)) d -= __ldg(col + b - 1) > __ldg(col + b);
  }
  d = warp_sum(d);
  if (lane_id() == 0 && d) atomicAdd((unsigned long long *)out, (unsigned long long)d);
}

// entries of the sorted row [b, e) below v
__device__ __forceinline__ int gc_below(const int *col, int64_t b, int64_t e, int v) {
  int64_t lo = b, hi = e;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(col + mid) < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (int)(lo - b);
}

// appends the lanes' vertices to a frontier and adds the arcs they will send along
// (no more than 2^25 a row, so that 32 of them fit: the sum is only compared with
// what one CTA takes)
__device__ __forceinline__ void gc_append(bool ready, int v, int arcs, int *q, gc_next_t *next) {
  const unsigned mask = __ballot_sync(FULL, ready);
  if (!mask) return;
  const int sum = __reduce_add_sync(FULL, ready ? MIN(arcs, 1 << 25) : 0);
  if (ready && arcs >= GC_LONG) next->longs = 1;
  int base = 0;
  if (lane_id() == 0) {
    base = atomicAdd(&next->size, __popc(mask));
    atomicAdd(&next->arcs, (unsigned long long)sum);
  }
  base = __shfl_sync(FULL, base, 0);
  if (ready) q[base + __popc(mask & ((1u << lane_id()) - 1u))] = v;
}

// cuts a row into pieces; every lane of the warp calls it
__device__ __forceinline__ void gc_cut(int64_t st, int lw, gc_piece_t *piece, int *pieces) {
  const int np = (lw + GC_PIECE - 1) / GC_PIECE;
  int base = 0;
  if (lane_id() == 0) base = atomicAdd(pieces, np);
  base = __shfl_sync(FULL, base, 0);
  for (int k = lane_id(); k < np; k += 32)
    piece[base + k] = gc_piece_t{st + (int64_t)k * GC_PIECE, MIN(GC_PIECE, lw - k * GC_PIECE)};
}

// wait: uncoloured larger in-neighbours per vertex; low: smaller
// out-neighbours; q: two frontiers of n.  A frontier lists only vertices that
// have smaller neighbours.  The last level that sends arcs settles a vertex
// that sends none, so the colour at which the frontier is empty is the largest.  first = 0: continue at S->at (the
// barrier words and the grid's frontier sizes zeroed again).
__global__ void __launch_bounds__(GC_THREADS, 1)
    k_gc_dag(device_graph_t<CSR, Empty> g, int *wait, int *low, int *colour, int *q0, int *q1, gc_piece_t *piece,
             gc_state_t *S, int first, unsigned long long budget_ns) {
  __shared__ int s_v[2][GC_SMALL_VERTICES];      // small frontier: vertex,
  __shared__ int s_low[2][GC_SMALL_VERTICES];    // its smaller neighbours
  __shared__ int64_t s_st[2][GC_SMALL_VERTICES];  // and where its row starts
  __shared__ int s_end[GC_SMALL_VERTICES], s_tmp[33];  // where each vertex's arcs end in the level's
  __shared__ int s_n[3], s_arcs[3], s_long;
  int *const q[2] = {q0, q1};
  const int lane = lane_id(), w = warp_id();
  const int64_t n = g.nvertexs;
  const int64_t nwarps = (int64_t)gridDim.x * (GC_THREADS / 32);
  const int64_t gw = (int64_t)blockIdx.x * (GC_THREADS / 32) + w;
  unsigned gen = 0;
  auto barrier = [&] { return grid_barrier(S->bar, S->bar + 1, S->bar + 2, gen, budget_ns); };
  // the same in every CTA: the frontier's colour, size and arcs, grid-wide
  // levels so far, hand-overs so far
  int L = 1, F = 0, M = 0, H = 0;
  unsigned long long A = 0;
  bool longs = false;  // the frontier has long rows
  unsigned done = 0;   // vertices this thread coloured
  int status = 0, ran = 0;
  bool okk = true;
  auto take = [&](const gc_next_t &next) {
    const int4 w = __ldcg((const int4 *)&next);
    A = (unsigned)w.x | (unsigned long long)(unsigned)w.y << 32;
    F = w.z;
    longs = w.w != 0;
  };
  if (first) {
    for (int64_t b = gw * 32; b < n; b += nwarps * 32) {
      const int v = (int)b + lane;
      bool ready = false;
      int lw = 0;
      if (v < n) {
        const int64_t st = __ldg(g.dg_row_off + v), en = __ldg(g.dg_row_off + v + 1);
        lw = gc_below(g.dg_adj_list, st, en, v);
        int wt = (int)(en - st) - lw;
        if (g.directed) {
          const int64_t rs = __ldg(g.dgr_row_off + v), re = __ldg(g.dgr_row_off + v + 1);
          wt = (int)(re - rs) - gc_below(g.dgr_adj_list, rs, re, v);
        }
        low[v] = lw;
        wait[v] = wt;
        ready = wt == 0;
        colour[v] = ready ? 1 : -1;
        done += ready;
      }
      gc_append(ready && lw > 0, v, lw, q[L & 1], &S->next[0]);
    }
    okk = barrier();
    take(S->next[0]);
  } else {
    L = S->at.level, F = S->at.size, A = S->at.arcs, longs = S->at.longs;
  }
  while (okk) {
    if (F == 0) break;
    if (ran >= GC_LAUNCH_LEVELS) {
      status = 1;
      break;
    }
    if (F <= GC_SMALL_VERTICES && A <= GC_SMALL_ARCS) {
      // CTA 0 alone, until the frontier empties or outgrows it
      if (blockIdx.x == 0) {
        int c = 0, nf = F, na, l = L;
        for (int i = threadIdx.x; i < nf; i += GC_THREADS) {
          const int v = __ldcg(q[L & 1] + i);
          s_v[0][i] = v;
          s_low[0][i] = __ldcg(low + v);
          s_st[0][i] = __ldg(g.dg_row_off + v);
        }
        if (threadIdx.x < 3) s_n[threadIdx.x] = s_arcs[threadIdx.x] = 0;
        if (threadIdx.x == 0) s_long = 0;
        __syncthreads();
        for (;;) {
          const int slot = l % 3;
          if (threadIdx.x == 0) s_n[(l + 1) % 3] = s_arcs[(l + 1) % 3] = 0;  // last read a level ago
          int total;
          const int lw = (int)threadIdx.x < nf ? s_low[c][threadIdx.x] : 0;
          const int ex = block_exclusive_scan(lw, s_tmp, &total);
          if ((int)threadIdx.x < nf) s_end[threadIdx.x] = ex + lw;
          __syncthreads();
          // consecutive arcs to a thread, all of them in flight
          const int per = (total + GC_THREADS - 1) / GC_THREADS, e0 = (int)threadIdx.x * per;
          int u[GC_ROWS], left[GC_ROWS];
          if (e0 < total) {
            int id = upper_bound(s_end, nf, e0);
            int64_t row = s_st[c][id] - (id ? s_end[id - 1] : 0);
#pragma unroll
            for (int k = 0; k < GC_ROWS; ++k) {
              u[k] = -1;
              if (k < per && e0 + k < total) {
                if (e0 + k >= s_end[id]) row = s_st[c][id + 1] - s_end[id], ++id;
                u[k] = __ldg(g.dg_adj_list + row + e0 + k);
              }
            }
#pragma unroll
            for (int k = 0; k < GC_ROWS; ++k) left[k] = u[k] >= 0 ? atomicSub(wait + u[k], 1) : 0;
#pragma unroll
            for (int k = 0; k < GC_ROWS; ++k) {
              if (left[k] != 1) continue;
              colour[u[k]] = l + 1;
              ++done;
              const int lu = __ldcg(low + u[k]);
              if (lu == 0) continue;
              const int at = atomicAdd(&s_n[slot], 1);
              atomicAdd(&s_arcs[slot], MIN(lu, GC_SMALL_ARCS + 1));
              if (lu >= GC_LONG) s_long = 1;
              if (at < GC_SMALL_VERTICES) {
                s_v[c ^ 1][at] = u[k];
                s_low[c ^ 1][at] = lu;
                s_st[c ^ 1][at] = __ldg(g.dg_row_off + u[k]);
              } else {
                q[(l + 1) & 1][at] = u[k];  // leaves shared memory after this level
              }
            }
          }
          __syncthreads();
          nf = s_n[slot];
          na = s_arcs[slot];
          ++l;
          c ^= 1;
          if (nf == 0 || nf > GC_SMALL_VERTICES || na > GC_SMALL_ARCS || l - L >= GC_SMALL_LEVELS) break;
        }
        for (int i = threadIdx.x; i < MIN(nf, GC_SMALL_VERTICES); i += GC_THREADS) q[l & 1][i] = s_v[c][i];
        if (threadIdx.x == 0) S->pub[H & 1] = gc_front_t{(unsigned)na, nf, l, s_long};
      }
      okk = barrier();
      const int4 w = __ldcg((const int4 *)&S->pub[H & 1]);
      const gc_front_t p{(unsigned)w.x, w.y, w.z, w.w};
      ran += p.level - L;
      L = p.level, F = p.size, A = p.arcs, longs = p.longs;
      ++H;
      continue;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      S->next[(M + 2) % 3] = gc_next_t{0, 0, 0};
      S->pieces[(M + 2) % 3] = 0;
    }
    // GC_BATCH arcs of a lane in flight, each the column of a vertex of this level
    auto arcs = [&](const int64_t (&e)[GC_BATCH], const bool (&valid)[GC_BATCH]) {
      int u[GC_BATCH], lu[GC_BATCH];
      bool ready[GC_BATCH];
#pragma unroll
      for (int k = 0; k < GC_BATCH; ++k) u[k] = valid[k] ? __ldg(g.dg_adj_list + e[k]) : -1;
#pragma unroll
      for (int k = 0; k < GC_BATCH; ++k) ready[k] = u[k] >= 0 && atomicSub(wait + u[k], 1) == 1;
#pragma unroll
      for (int k = 0; k < GC_BATCH; ++k) lu[k] = ready[k] ? __ldcg(low + u[k]) : 0;
#pragma unroll
      for (int k = 0; k < GC_BATCH; ++k) {
        if (ready[k]) {
          colour[u[k]] = L + 1;
          ++done;
        }
        gc_append(lu[k] > 0, u[k], lu[k], q[(L + 1) & 1], &S->next[(M + 1) % 3]);
      }
    };
    // the frontier's rows, then, once all of them are listed, the pieces of the long ones
    int rows = F;
    for (int cut = 0;; cut = 1) {
      auto row = [&](int64_t i, int64_t &st, int &lw) {
        if (cut) {
          const gc_piece_t p = piece[i];
          st = p.beg, lw = p.len;
        } else {
          const int v = __ldcg(q[L & 1] + i);
          st = __ldg(g.dg_row_off + v), lw = __ldcg(low + v);
        }
      };
      if (rows <= nwarps) {  // several warps to a row
        const int per = (int)(nwarps / rows);
        if (gw / per < rows) {
          int64_t st;
          int lw;
          row(gw / per, st, lw);
          if (lw / GC_LONG >= per) {
            if (gw % per == 0) gc_cut(st, lw, piece, &S->pieces[M % 3]);
            lw = 0;
          }
          for (int k0 = (int)(gw % per) * 32; k0 < lw; k0 += per * 32 * GC_BATCH) {
            int64_t e[GC_BATCH];
            bool valid[GC_BATCH];
#pragma unroll
            for (int k = 0; k < GC_BATCH; ++k) {
              const int at = k0 + per * 32 * k + lane;
              e[k] = st + at;
              valid[k] = at < lw;
            }
            arcs(e, valid);
          }
        }
      } else {  // a warp takes `per` rows and walks their arcs 32 at a time
        const int per = (int)MIN((int64_t)32, (rows + nwarps - 1) / nwarps);
        for (int64_t b = gw * per; b < rows; b += nwarps * per) {
          int lw = 0;
          int64_t st = 0;
          if (lane < per && b + lane < rows) row(b + lane, st, lw);
          if (longs)
            for (unsigned m = __ballot_sync(FULL, lw >= GC_LONG); m; m &= m - 1) {
              const int src = __ffs(m) - 1;
              gc_cut(__shfl_sync(FULL, st, src), __shfl_sync(FULL, lw, src), piece, &S->pieces[M % 3]);
              if (lane == src) lw = 0;
            }
          const int incl = warp_inclusive_sum(lw);
          const int total = __shfl_sync(FULL, incl, 31);
          for (int e0 = 0; e0 < total; e0 += 32 * GC_BATCH) {
            int64_t e[GC_BATCH];
            bool valid[GC_BATCH];
#pragma unroll
            for (int k = 0; k < GC_BATCH; ++k) {
              const int at = e0 + 32 * k + lane;
              // the row that holds it: the first lane with incl > at
              int lo = 0;
#pragma unroll
              for (int s = 16; s > 0; s >>= 1) {
                const int x = __shfl_sync(FULL, incl, lo + s - 1);
                if (x <= at) lo += s;
              }
              const int before = __shfl_sync(FULL, incl - lw, lo & 31);
              e[k] = __shfl_sync(FULL, st, lo & 31) + (at - before);
              valid[k] = at < total;
            }
            arcs(e, valid);
          }
        }
      }
      if (!longs || cut) break;
      okk = barrier();
      rows = okk ? ((volatile int *)S->pieces)[M % 3] : 0;
      if (rows == 0) break;
    }
    okk = okk && barrier();
    ++M;
    take(S->next[M % 3]);
    ++L;
    ++ran;
  }
  done = __reduce_add_sync(FULL, done);
  if (lane == 0 && done) atomicAdd(&S->coloured, (unsigned long long)done);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S->at = gc_front_t{(unsigned)MIN(A, 0x7fffffffull), F, L, longs};
    S->status = okk ? status : 2;
  }
}

}  // namespace gsw
