/*
 * wave.cu — near-far SSSP by one CTA or a group of CTAs per query.
 *
 * Replaces, for thin wave fronts and for batches of many queries, the
 * worklist of the reference (ads_int/wl.h:133-1972) and its relaxation
 * (ads_int/kernel.cu:30-128).  A road network's wave front is a chain of a
 * thousand or more dependent steps; what a step costs is its memory round
 * trips and its barrier, not its bytes.  Here a CTA runs the chain alone: its
 * frontier lives in shared memory, a step's barrier is bar.sync, and nothing is
 * counted, published or claimed through HBM.  A group of CTAs (a CTA per SM for
 * a plain solve) shares a query: each runs several steps on its own entries,
 * then they exchange what is left through lists and 16-byte notes in HBM.
 * (A cluster of 16 CTAs with lists in distributed shared memory was slower: a
 * barrier.cluster with release costs about 3,500 cycles, and 16 SMs are few.)
 * Many CTAs or groups run side by side in a batch: single CTAs draw queries
 * from a shared counter, largest first; groups get shares of equal work.
 *
 * A step pops the frontier's entries (v, d), drops those that a smaller
 * distance has superseded, relaxes the rows and keeps the improvements: those
 * below the near threshold T are the next frontier, the others go to the
 * CTA's far list.  When the frontier is empty, or small while far entries
 * wait, T moves up and the far list is split again (stale entries dropped,
 * the rest kept).  Any sequence of thresholds is label-correcting, so the
 * distances are the fixed point that every other engine reaches.
 *
 * An improvement is pushed by the one thread whose atomicMin lowered the
 * distance: steps are in lock step, so pushing on the gathered value alone
 * (as the asynchronous engine does) would push a vertex once for each of its
 * equal paths, and those copies multiply from step to step.
 *
 * What bounds it: the chain of memory round trips of a hop (row bounds, edges,
 * atomicMin and its answer: about 3,400 cycles with the push and the barrier,
 * in a group; a load from L2 takes 310 to 460 cycles, an atomic 510 to 870),
 * and, where a CTA has hundreds of entries, its rate of scattered requests
 * (one sector a cycle and SM, an atomic two cycles).  Hence: the row bounds of
 * an improvement are prefetched while its atomicMin is on its way, four lanes
 * share a vertex so that a row comes with one request, and small hops skip the
 * filtering load of the distance before the atomic.  A group's CTAs run several
 * hops on their own entries between two exchanges, which cost about 6,000
 * cycles: neighbouring entries stay together, so few of these hops relax from a
 * distance that another CTA is about to lower.
 *
 * Measured (B200, automatic knobs, one call with its copy and wait, before ->
 * now; the kernel alone in brackets, three graphs): 4096^2 road-like grid 261-310
 * -> 17.9-19.9 ms (17.3-19.8); 517 x 301 road 16-21 -> 1.1-1.3 ms (0.85-1.2); 128
 * grids x 16 sources in one batch 97.7 -> 7.2 ms; 60 sources on a 257 x 255 road 4.7
 * -> 1.6 ms; R-MAT 16 0.87 -> 0.37-0.42 ms (0.28); ER 4,001 x 8 0.57 -> 0.16 ms
 * (0.08-0.10).
 *
 * Graphs with long rows (POOL): rows are cut into pieces that exchanges deal
 * out, a CTA pools the edges of its entries over its threads, and on large
 * graphs light and heavy edges are relaxed apart: heavy edges (which cannot
 * land in the bucket that is being settled) once per settled vertex, when the
 * frontier has run low.  R-MAT 20 relaxes 1.0 to 1.3 times its edges so, 3.5 to
 * 4 times with whole rows; 0.85 ms against 1.2, and 1.8 on the phase engine.
 * From some 17 million edges on, heavy hops that would relax more edges than the
 * in-edges of the vertices above T are pulls (WV_PULL): R-MAT 22 with float
 * weights 3.9 -> 3.6 ms with its copies, a batch of 8 R-MATs 21.2 -> 19.1.
 * A full hop is bound by scattered requests (gathers 1,900, atomics 2,000, row
 * searches and edge loads 2,500, pushes 1,400 cycles for 4,096 edges of an SM),
 * a small one by its round trips.
 *
 * The lists cannot grow: an overflow ends the launch with WV_ERR_OVERFLOW and
 * the host solves on another engine.
 */
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>

#include "../../include/adds.h"
#include "adds_internal.h"
#include "wave_internal.h"

namespace adds_wave {

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

/* what the CTAs of a group tell each other at an exchange */
struct __align__(16) Note {
  unsigned near_cnt, far_cnt, far_min, stop; /* stop: errors, WV_SETTLED     */
};

/* a hop's pushes: entries of the next frontier, far entries added, error.
 * Three of them rotate: the one a hop reads, the one it fills, and the one it
 * clears for the next, so that a hop needs one barrier. */
struct __align__(16) Ctr {
  unsigned near_cnt, far_new, stop;
  unsigned cut;     /* a long row became pieces                               */
  unsigned set_new; /* settled entries added                                  */
  unsigned pad[3];
};

#define PULL_V 4u /* vertices a thread takes per chunk of a pull              */

template <int BLOCK, int NS, int PL>
struct WSmem {
  uint2 nb[2][NS];  /* frontier entries (v, d): this hop's, the next          */
  Ctr ctr[3];
  Note tot;         /* the group's totals                                     */
  unsigned far_max; /* the longest far list of a CTA                          */
  unsigned kept;    /* far entries a split has kept                           */
  unsigned fmin;    /* the smallest distance among them                       */
  unsigned q, r0;
  unsigned pre[WV_MAX_GROUP]; /* inclusive frontier counts of the CTAs        */
  /* POOL: the rows being relaxed by the whole CTA, and their edge offsets    */
  static constexpr int PB = PL == 2 ? PULL_V * BLOCK : (PL == 1 ? BLOCK : 1);
  unsigned it_r0[PB], it_d[PB], it_off[PB], wsum[32];
  /* POOL with in-edges: the settled entries' heavy edges and in-edges (an
   * entry that settles twice counts twice), and their smallest distance; the
   * group's totals                                                           */
  unsigned long long heavy, into, t_heavy, t_into;
  unsigned smin, t_smin, t_set, gsize;
};

/* lists of one CTA in HBM */
struct Lists {
  uint2 *over;      /* frontier entries past the shared ones: two areas       */
  uint2 *far;
  uint2 *set;       /* settled entries (light/heavy split)                    */
  unsigned ncap, fcap, scap;
};

template <bool FLT>
__device__ __forceinline__ unsigned add_word(unsigned d, unsigned w) {
  return FLT ? __float_as_uint(__fadd_rn(__uint_as_float(d), __uint_as_float(w))) : d + w;
}

/* threshold word of distance word d plus delta; never below d + 1, so that a
 * threshold taken from an entry always admits it */
template <bool FLT>
__device__ __forceinline__ unsigned raise_word(unsigned d, float delta) {
  unsigned t;
  if (FLT) {
    t = __float_as_uint(__fadd_rn(__uint_as_float(d), delta));
  } else {
    const double x = (double)d + (double)delta;
    t = x < 4294967295.0 ? (unsigned)x : 0xFFFFFFFFu;
  }
  return t > d ? t : d + (d != 0xFFFFFFFFu);
}

/* a note in one 16-byte access */
__device__ __forceinline__ void st_note(ulonglong2 *p, unsigned a, unsigned b, unsigned c,
                                        unsigned d) {
  const unsigned long long lo = a | ((unsigned long long)b << 32);
  const unsigned long long hi = c | ((unsigned long long)d << 32);
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
               "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ uint4 ld_note(const ulonglong2 *p) {
  unsigned long long lo, hi;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}

/* GRP: several CTAs per query.  POOL: a CTA pools the edges of its entries
 * over all its threads (graphs whose rows differ much in length); without it
 * each warp relaxes its own entries.  PULL: heavy hops may be pulls (PL 0: none
 * of these, 1: POOL, 2: both; the code alone costs the pooled hop 5 % in
 * registers). */
template <bool FLT, int BLOCK, int NS, bool GRP, int PL>
struct Wave {
  static constexpr bool POOL = PL >= 1, PULL = PL == 2;
  using Smem = WSmem<BLOCK, NS, PL>;

  /* one thread's state over a query; all but the counts is uniform */
  struct State {
    Lists L;
    const unsigned *row;
    const uint2 *edges;
    const unsigned *first; /* long rows: a row's first piece, the pieces       */
    const uint4 *piece;
    const unsigned *split; /* light edges at the start of each row, or null    */
    const unsigned *trow;  /* in-edges, or null: heavy hops may be pulls        */
    unsigned *dist;
    unsigned n, np;
    unsigned T;    /* near threshold (distance word)                          */
    unsigned cur;  /* frontier buffer being read                              */
    unsigned ci;   /* counter of that frontier                                */
    unsigned F;    /* far entries of this CTA                                 */
    unsigned H;    /* settled entries of this CTA                             */
    unsigned npush, nstale;
    unsigned long long nedge;
  };
  static constexpr unsigned SUB = BLOCK < 256 ? BLOCK : 256; /* a part of a pooled CTA */
  static __device__ __forceinline__ void bar_part(unsigned part) {
    asm volatile("bar.sync %0, %1;" ::"r"(part + 1u), "r"(SUB) : "memory");
  }
  static __device__ __forceinline__ unsigned next3(unsigned i) { return i == 2u ? 0u : i + 1u; }

  static __device__ __forceinline__ uint2 entry(const Smem &S, const State &w, unsigned i) {
    return i < NS ? S.nb[w.cur][i] : __ldcg(w.L.over + (size_t)w.cur * w.L.ncap + (i - NS));
  }
  static __device__ __forceinline__ void put(Smem &S, const State &w, unsigned buf, unsigned i,
                                             uint2 e) {
    if (i < NS) S.nb[buf][i] = e;
    else if (i - NS < w.L.ncap) __stcg(w.L.over + (size_t)buf * w.L.ncap + (i - NS), e);
  }

  /* Appends the lanes' improvements (v, nd) in keep to frontier buffer buf and
   * the far list: one reservation per list and warp.  Returns what lane 0 is
   * to count. */
  template <int U>
  static __device__ __forceinline__ unsigned push(Smem &S, const State &w, Ctr &C, unsigned buf,
                                                  const unsigned (&v)[U], const unsigned (&nd)[U],
                                                  unsigned keep) {
    const unsigned lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    unsigned bn[U], bf[U], cn = 0, cf = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool p = (keep >> u) & 1u, nr = nd[u] < w.T;
      bn[u] = __ballot_sync(0xFFFFFFFFu, p && nr);
      bf[u] = __ballot_sync(0xFFFFFFFFu, p && !nr);
      cn += __popc(bn[u]);
      cf += __popc(bf[u]);
    }
    if ((cn | cf) == 0u) return 0u;
    unsigned at = 0;
    if (lane < 2u) at = atomicAdd(lane ? &C.far_new : &C.near_cnt, lane ? cf : cn);
    unsigned pn = __shfl_sync(0xFFFFFFFFu, at, 0);
    unsigned pf = __shfl_sync(0xFFFFFFFFu, at, 1) + w.F;
    if (pn + cn > NS + w.L.ncap || pf + cf > w.L.fcap) C.stop = WV_ERR_OVERFLOW;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint2 e = make_uint2(v[u], nd[u]);
      if ((bn[u] >> lane) & 1u) put(S, w, buf, pn + __popc(bn[u] & lt), e);
      if ((bf[u] >> lane) & 1u) {
        const unsigned i = pf + __popc(bf[u] & lt);
        if (i < w.L.fcap) __stcg(w.L.far + i, e);
      }
      pn += __popc(bn[u]);
      pf += __popc(bf[u]);
    }
    return lane == 0u ? cn + cf : 0u;
  }

  /* Relaxes the edges ed (those in msk) of each lane from distance words dd
   * and pushes the improvements: one reservation per list and warp. */
  template <int U>
  static __device__ __forceinline__ void relax(Smem &S, State &w, const uint2 (&ed)[U],
                                               const unsigned (&dd)[U], unsigned msk,
                                               bool direct = false) {
    unsigned nd[U], cur[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      nd[u] = add_word<FLT>(dd[u], ed[u].y);
      cur[u] = 0u;
      if ((msk >> u) & 1u) cur[u] = direct ? 0xFFFFFFFFu : __ldcg(w.dist + ed[u].x);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) { /* absent edges hold cur 0: never below */
      if (nd[u] < cur[u]) {
        cur[u] = atomicMin(w.dist + ed[u].x, nd[u]);
        /* the row bounds are wanted as soon as the entry is popped */
        if (GRP && nd[u] < w.T)
          asm volatile("prefetch.global.L1 [%0];" ::"l"(w.row + ed[u].x));
      } else {
        cur[u] = 0u;
      }
    }
    unsigned keep = 0, v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      v[u] = ed[u].x;
      if (nd[u] < cur[u]) keep |= 1u << u;
    }
    w.npush += push<U>(S, w, S.ctr[next3(w.ci)], w.cur ^ 1u, v, nd, keep);
  }

  /* a lane's entry: its row (or its piece of a long row: ids from n up), and
   * whether its distance is still the vertex's */
  static __device__ __forceinline__ void load(const State &w, uint2 x, bool in, unsigned &r0,
                                              unsigned &deg, bool &live) {
    r0 = deg = 0u;
    live = false;
    if (in) {
      unsigned v = x.x;
      if (v < w.n) {
        r0 = __ldg(w.row + v);
        deg = __ldg(w.row + v + 1) - r0;
      } else {
        const uint4 c = __ldg(w.piece + (v - w.n));
        v = c.x;
        r0 = c.y;
        deg = c.z;
      }
      live = __ldcg(w.dist + v) == x.y;
    }
  }

  /* A long row becomes pieces of WV_PIECE edges in the next frontier, which
   * an exchange deals out over the group (one warp on a row of thousands of
   * edges would hold up the hop). */
  static __device__ __forceinline__ void cut(Smem &S, State &w, uint2 x, unsigned deg) {
    Ctr &C = S.ctr[next3(w.ci)];
    const unsigned k = (deg + WV_PIECE - 1u) / WV_PIECE, c0 = w.n + __ldg(w.first + x.x);
    const unsigned at = atomicAdd(&C.near_cnt, k);
    if (at + k > NS + w.L.ncap) C.stop = WV_ERR_OVERFLOW;
    C.cut = 1u;
    for (unsigned j = 0; j < k; ++j) put(S, w, w.cur ^ 1u, at + j, make_uint2(c0 + j, x.y));
  }

  /* The edges of up to 32 entries (one a lane) spread over the warp: 32
   * neighbouring edges per load, a lane's row found by a search over the
   * row offsets. */
  static __device__ __forceinline__ void spread(Smem &S, State &w, uint2 x, unsigned r0,
                                                unsigned deg) {
    constexpr int U = 4;
    const unsigned lane = threadIdx.x & 31u;
    unsigned off = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xFFFFFFFFu, off, o);
      if (lane >= (unsigned)o) off += y;
    }
    const unsigned E = __shfl_sync(0xFFFFFFFFu, off, 31);
    off -= deg;
    if (lane == 0) w.nedge += E;
    for (unsigned e0 = 0; e0 < E; e0 += 32u * U) {
      uint2 e[U];
      unsigned dd[U], msk = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned k = e0 + u * 32u + lane;
        unsigned j = 0;
#pragma unroll
        for (int b = 16; b > 0; b >>= 1) {
          const unsigned o = __shfl_sync(0xFFFFFFFFu, off, j + b);
          if (o <= k) j += b;
        }
        const unsigned ro = __shfl_sync(0xFFFFFFFFu, r0, j);
        const unsigned oo = __shfl_sync(0xFFFFFFFFu, off, j);
        dd[u] = __shfl_sync(0xFFFFFFFFu, x.y, j);
        e[u] = make_uint2(0u, 0u);
        if (k < E) {
          e[u] = __ldg(w.edges + ro + (k - oo));
          msk |= 1u << u;
        }
      }
      relax<U>(S, w, e, dd, msk);
    }
  }

  /* A pooled hop's entry.  With the light/heavy split (rows sorted by weight)
   * an id below n is a vertex whose light edges are wanted, then come the light
   * pieces of long rows, their heavy pieces, and vertices whose heavy edges
   * are.  set: the vertex joins the settled list, for its heavy edges.  Rows
   * longer than a piece are cut here, deg is 0 for them. */
  static __device__ __forceinline__ void load_pool(Smem &S, State &w, uint2 x, bool in,
                                                   unsigned &r0, unsigned &deg, bool &set) {
    r0 = deg = 0u;
    set = false;
    if (!in) return;
    unsigned v = x.x, j0 = 0, len = 0;
    const bool whole = v < w.n || v >= w.n + 2u * w.np;
    bool heavy = v >= w.n + w.np;
    if (whole) {
      if (heavy) v -= w.n + 2u * w.np;
      r0 = __ldg(w.row + v);
      len = __ldg(w.row + v + 1) - r0;
      deg = len;
      if (w.split) {
        const unsigned nl = __ldg(w.split + v);
        set = !heavy && nl < len;
        j0 = heavy ? nl / WV_PIECE : 0u;
        deg = heavy ? len - nl : nl;
        len = heavy ? len : nl; /* pieces from j0 on reach as far as this */
        if (heavy) r0 += nl;
      }
    } else {
      const uint4 c = __ldg(w.piece + (v - w.n - (heavy ? w.np : 0u)));
      v = c.x;
      r0 = c.y;
      deg = c.z;
      if (w.split) {
        const unsigned off = c.y - __ldg(w.row + v), nl = __ldg(w.split + v);
        if (heavy && nl > off) {
          r0 += nl - off;
          deg -= nl - off;
        } else if (!heavy) {
          deg = min(deg, nl - off);
        }
      }
    }
    if (__ldcg(w.dist + v) != x.y) {
      ++w.nstale;
      deg = 0u;
      set = false;
    } else if (whole && deg > WV_PIECE) {
      Ctr &C = S.ctr[next3(w.ci)];
      const unsigned j1 = (len + WV_PIECE - 1u) / WV_PIECE, k = j1 - j0;
      const unsigned c0 = w.n + (heavy ? w.np : 0u) + __ldg(w.first + v) + j0;
      const unsigned at = atomicAdd(&C.near_cnt, k);
      if (at + k > NS + w.L.ncap) C.stop = WV_ERR_OVERFLOW;
      C.cut = 1u;
      for (unsigned j = 0; j < k; ++j) put(S, w, w.cur ^ 1u, at + j, make_uint2(c0 + j, x.y));
      deg = 0u;
    }
  }

  /* Ends a bucket: the settled entries that are still current become frontier
   * entries for their heavy edges.  Uniform over the CTA. */
  static __device__ void unsettle(Smem &S, State &w) {
    const unsigned tid = threadIdx.x, lane = tid & 31u, lt = (1u << lane) - 1u;
    Ctr &C = S.ctr[w.ci];
    for (unsigned i0 = 0; i0 < w.H; i0 += BLOCK) {
      const bool have = i0 + tid < w.H;
      const uint2 x = have ? __ldcg(w.L.set + i0 + tid) : make_uint2(0u, 0u);
      const bool in = have && __ldcg(w.dist + x.x) == x.y;
      const unsigned b = __ballot_sync(0xFFFFFFFFu, in);
      if (b == 0u) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&C.near_cnt, (unsigned)__popc(b));
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      if (at + __popc(b) > NS + w.L.ncap) C.stop = WV_ERR_OVERFLOW;
      if (in) put(S, w, w.cur, at + __popc(b & lt), make_uint2(x.x + w.n + 2u * w.np, x.y));
    }
    w.H = 0u;
    __syncthreads();
  }

  /* The heavy edges of the settled vertices taken from the other side: every
   * vertex whose distance lies above floor -- the only ones they can improve,
   * floor being the smallest settled distance plus the smallest heavy weight --
   * takes the minimum over its in-edges.  Every candidate is a path's length, a
   * vertex is written by its thread only, and an improvement that a neighbour
   * misses in this hop reaches it when the improved vertex is popped.
   * Improvements join the frontier that is waiting, and the far list.  For
   * large buckets of graphs whose hubs settle early: R-MAT 22 relaxes 1.3 times
   * its edges without, 0.54 with (1.8 against 1.6 ms; float 2.05 against 1.92). */
  static __device__ __noinline__ unsigned pull(Smem &S, State w, const uint2 *tedges,
                                               unsigned floor, unsigned &edges) {
    constexpr int U = 4, V = PULL_V;
    const unsigned part = threadIdx.x / SUB, tid = threadIdx.x % SUB, lane = tid & 31u;
    const unsigned warp = tid >> 5, nparts = BLOCK / SUB;
    const unsigned G = S.gsize, rank = blockIdx.x % G;
    unsigned *const it_r0 = S.it_r0 + part * SUB * V, *const it_b = S.it_d + part * SUB * V;
    unsigned *const it_off = S.it_off + part * SUB * V, *const wsum = S.wsum + part * (SUB / 32u);
    const bool vec = ((reinterpret_cast<unsigned long long>(w.dist) |
                       reinterpret_cast<unsigned long long>(w.trow)) & 15ull) == 0ull;
    unsigned npush = 0, nedge = 0;
    const unsigned long long step = (unsigned long long)G * nparts * SUB * V;
    for (unsigned long long c0 = ((unsigned long long)rank * nparts + part) * SUB * V; c0 < w.n;
         c0 += step) {
      const unsigned long long v0 = c0 + tid * V;
      unsigned d[V], rb[V + 1];
      if (vec && v0 + V <= w.n) {
        const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(w.dist + v0));
        const uint4 r = __ldg(reinterpret_cast<const uint4 *>(w.trow + v0));
        d[0] = x.x; d[1] = x.y; d[2] = x.z; d[3] = x.w;
        rb[0] = r.x; rb[1] = r.y; rb[2] = r.z; rb[3] = r.w;
        rb[4] = __ldg(w.trow + v0 + 4);
      } else {
#pragma unroll
        for (int j = 0; j <= V; ++j) {
          if (j < V) d[j] = v0 + j < w.n ? __ldcg(w.dist + v0 + j) : 0u;
          rb[j] = v0 + j <= w.n ? __ldg(w.trow + v0 + j) : 0u;
        }
      }
      unsigned sum = 0;
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (v0 + j < w.n && d[j] > floor) sum += rb[j + 1] - rb[j];
      unsigned off = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, off, o);
        if (lane >= (unsigned)o) off += y;
      }
      if (lane == 31u) wsum[warp] = off;
      bar_part(part);
      unsigned ws = lane < SUB / 32u ? wsum[lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, ws, o);
        if (lane >= (unsigned)o) ws += y;
      }
      const unsigned E = __shfl_sync(0xFFFFFFFFu, ws, 31);
      const unsigned wb = __shfl_sync(0xFFFFFFFFu, ws, (warp + 31u) & 31u);
      unsigned at = off - sum + (warp ? wb : 0u);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const unsigned i = tid * V + j;
        it_r0[i] = rb[j];
        it_b[i] = d[j]; /* the best so far */
        it_off[i] = at;
        if (v0 + j < w.n && d[j] > floor) at += rb[j + 1] - rb[j];
      }
      nedge += sum;
      bar_part(part);
      const unsigned k = SUB * V;
      const unsigned run = ((E + SUB / 32u - 1u) / (SUB / 32u) + 31u) & ~31u;
      const unsigned re = min(E, (warp + 1u) * run);
      unsigned lo = 0, fin = 0, at0 = 0;
      for (unsigned e0 = warp * run; e0 < re; e0 += 32u * U) {
        uint2 e[U];
        unsigned it[U], cur[U], msk = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned j = e0 + u * 32u + lane;
          e[u] = make_uint2(0u, 0u);
          if (j < re) {
            if (j >= fin) {
              unsigned st = 1u;
              while (lo + st < k && it_off[lo + st] <= j) {
                lo += st;
                st <<= 1;
              }
              unsigned hi = min(lo + st, k) - 1u;
              while (lo < hi) {
                const unsigned mid = (lo + hi + 1u) >> 1;
                if (it_off[mid] <= j) lo = mid; else hi = mid - 1u;
              }
              fin = lo + 1u < k ? it_off[lo + 1u] : E;
              at0 = it_r0[lo] - it_off[lo];
            }
            e[u] = __ldg(tedges + (at0 + j));
            msk |= 1u << u;
          }
          it[u] = lo;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = ((msk >> u) & 1u) ? __ldcg(w.dist + e[u].x) : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned cand = add_word<FLT>(cur[u], e[u].y); /* INF + w improves nothing */
          if (((msk >> u) & 1u) && cand < it_b[it[u]]) atomicMin(&it_b[it[u]], cand);
        }
      }
      bar_part(part);
      unsigned v[V], nd[V], keep = 0;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        v[j] = (unsigned)(v0 + j);
        nd[j] = it_b[tid * V + j];
        if (v0 + j < w.n && nd[j] < d[j]) {
          keep |= 1u << j;
          __stcg(w.dist + v[j], nd[j]);
        }
      }
      npush += push<V>(S, w, S.ctr[w.ci], w.cur, v, nd, keep);
      bar_part(part);
    }
    edges += nedge;
    return npush;
  }

  /* A hop whose edges are pooled: SUB threads take every (BLOCK / SUB)th entry,
   * scan the row lengths of SUB entries at a time, and every warp walks 32 x U
   * neighbouring edges at a time.  The parts of a CTA meet only at the hop's
   * end, so that one loads entries while another relaxes edges (256 mixed queries 21.9 ms as one part, 21.2 in four). */
  static __device__ __forceinline__ void hop_pool(Smem &S, State &w, unsigned cnt) {
    constexpr int U = 4;
    constexpr unsigned PARTS = BLOCK / SUB;
    const unsigned part = threadIdx.x / SUB, tid = threadIdx.x % SUB, lane = tid & 31u;
    const unsigned warp = tid >> 5, lt = (1u << lane) - 1u, mine = cnt > part ? (cnt - part + PARTS - 1u) / PARTS : 0u;
    unsigned *const it_r0 = S.it_r0 + part * SUB, *const it_d = S.it_d + part * SUB;
    unsigned *const it_off = S.it_off + part * SUB, *const wsum = S.wsum + part * (SUB / 32u);
    if (threadIdx.x == 0) S.ctr[next3(next3(w.ci))] = Ctr{};
    for (unsigned i0 = 0; i0 < mine; i0 += SUB) {
      const bool in = i0 + tid < mine;
      const uint2 x = in ? entry(S, w, (i0 + tid) * PARTS + part) : make_uint2(0u, 0u);
      unsigned r0, deg;
      bool set;
      load_pool(S, w, x, in, r0, deg, set);
      const unsigned sb = __ballot_sync(0xFFFFFFFFu, set);
      if (sb) {
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&S.ctr[next3(w.ci)].set_new, (unsigned)__popc(sb));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + w.H + __popc(sb & lt);
        if (PULL && w.trow) { /* what a push and a pull of these heavy edges would read */
          unsigned hv = 0, in = 0;
          if (set) {
            hv = __ldg(w.row + x.x + 1) - __ldg(w.row + x.x) - __ldg(w.split + x.x);
            in = __ldg(w.trow + x.x + 1) - __ldg(w.trow + x.x);
          }
          hv = __reduce_add_sync(0xFFFFFFFFu, hv);
          in = __reduce_add_sync(0xFFFFFFFFu, in);
          const unsigned sm = __reduce_min_sync(0xFFFFFFFFu, set ? x.y : 0xFFFFFFFFu);
          if (lane == 0) {
            atomicAdd(&S.heavy, (unsigned long long)hv);
            atomicAdd(&S.into, (unsigned long long)in);
            atomicMin(&S.smin, sm);
          }
        }
        if (set) {
          if (at < w.L.scap) __stcg(w.L.set + at, x);
          else S.ctr[next3(w.ci)].stop = WV_ERR_OVERFLOW;
        }
      }
      unsigned off = deg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, off, o);
        if (lane >= (unsigned)o) off += y;
      }
      if (lane == 31u) wsum[warp] = off;
      it_r0[tid] = r0;
      it_d[tid] = x.y;
      bar_part(part);
      unsigned ws = lane < SUB / 32u ? wsum[lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, ws, o);
        if (lane >= (unsigned)o) ws += y;
      }
      const unsigned E = __shfl_sync(0xFFFFFFFFu, ws, 31);
      const unsigned wb = __shfl_sync(0xFFFFFFFFu, ws, (warp + 31u) & 31u);
      it_off[tid] = off - deg + (warp ? wb : 0u);
      w.nedge += deg;
      bar_part(part);
      const unsigned k = min((unsigned)SUB, mine - i0);
      /* each warp a run of neighbouring edges: a lane's next edge is 32 further,
       * so its row is at most a few items on */
      const unsigned run = ((E + SUB / 32u - 1u) / (SUB / 32u) + 31u) & ~31u;
      const unsigned re = min(E, (warp + 1u) * run);
      /* item of the lane's last edge (its edges only move forward), where the
       * item's edges end, and its row and distance */
      unsigned lo = 0, fin = 0, shift_r = 0, dcur = 0;
      for (unsigned e0 = warp * run; e0 < re; e0 += 32u * U) {
        uint2 e[U];
        unsigned dd[U], msk = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned j = e0 + u * 32u + lane;
          e[u] = make_uint2(0u, 0u);
          if (j < re) {
            if (j >= fin) {
              unsigned step = 1u;
              while (lo + step < k && it_off[lo + step] <= j) {
                lo += step;
                step <<= 1;
              }
              unsigned hi = min(lo + step, k) - 1u;
              while (lo < hi) {
                const unsigned mid = (lo + hi + 1u) >> 1;
                if (it_off[mid] <= j) lo = mid; else hi = mid - 1u;
              }
              fin = lo + 1u < k ? it_off[lo + 1u] : E;
              shift_r = it_r0[lo] - it_off[lo];
              dcur = it_d[lo];
            }
            e[u] = __ldg(w.edges + (shift_r + j));
            msk |= 1u << u;
          }
          dd[u] = dcur;
        }
        relax<U>(S, w, e, dd, msk);
      }
      bar_part(part); /* the pool is read */
    }
  }

  /* One hop: relaxes the rows of the cnt frontier entries into the next
   * frontier and the far list.  The caller's barrier ends it. */
  static __device__ __forceinline__ void hop(Smem &S, State &w, unsigned cnt) {
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) S.ctr[next3(next3(w.ci))] = Ctr{};
    /* few entries: eight a warp, four lanes each, rows of up to eight edges in
     * one round, so that every warp of the CTA has part of the hop */
    const bool few = cnt <= BLOCK / 4u;
    for (unsigned i0 = warp * (few ? 8u : 32u); i0 < cnt; i0 += BLOCK) {
      const unsigned i = i0 + (few ? lane >> 2 : lane);
      const bool in = i < cnt, first = !few || (lane & 3u) == 0u;
      const uint2 x = in ? entry(S, w, i) : make_uint2(0u, 0u);
      unsigned r0, deg;
      bool live;
      load(w, x, in, r0, deg, live);
      if (first && in && !live) ++w.nstale;
      if (deg > WV_PIECE && x.x < w.n) {
        if (live && first) cut(S, w, x, deg);
        deg = 0u;
      }
      if (GRP && few && __reduce_max_sync(0xFFFFFFFFu, deg) <= 8u) {
        uint2 e[2];
        const unsigned dd[2] = {x.y, x.y};
        unsigned msk = 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const unsigned k = u * 4u + (lane & 3u);
          e[u] = make_uint2(0u, 0u);
          if (k < deg) { /* read before it is known whether the entry is live */
            e[u] = __ldg(w.edges + r0 + k);
            msk |= 1u << u;
          }
        }
        if (!live) msk = 0;
        if (live && first) w.nedge += deg;
        relax<2>(S, w, e, dd, msk, true);
        continue;
      }
      if (!live) deg = 0u;
      const unsigned maxdeg = __reduce_max_sync(0xFFFFFFFFu, deg);
      if (maxdeg <= 8u) {
        /* short rows: four lanes to a vertex, eight vertices to a load, so
         * that a row's edges come with one request */
        if (first) w.nedge += deg;
        for (unsigned k0 = 0; k0 < maxdeg; k0 += 4u) {
          const unsigned k = k0 + (lane & 3u);
          if (few) {
            const uint2 e[1] = {k < deg ? __ldg(w.edges + r0 + k) : make_uint2(0u, 0u)};
            const unsigned dd[1] = {x.y};
            relax<1>(S, w, e, dd, k < deg ? 1u : 0u);
            continue;
          }
          uint2 e[4];
          unsigned dd[4], msk = 0;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int own = u * 8 + (int)(lane >> 2);
            const unsigned ro = __shfl_sync(0xFFFFFFFFu, r0, own);
            const unsigned dg = __shfl_sync(0xFFFFFFFFu, deg, own);
            dd[u] = __shfl_sync(0xFFFFFFFFu, x.y, own);
            e[u] = make_uint2(0u, 0u);
            if (k < dg) {
              e[u] = __ldg(w.edges + ro + k);
              msk |= 1u << u;
            }
          }
          relax<4>(S, w, e, dd, msk);
        }
      } else {
        spread(S, w, x, r0, first ? deg : 0u);
      }
    }
  }

  /* Moves T up and splits this CTA's far list against it: entries below join
   * the frontier, stale ones are dropped, the others are packed in place (a
   * tile is read before any of it is written over).  Uniform over the CTA;
   * the counter's frontier count and w.F are current afterwards. */
  static __device__ void split(Smem &S, State &w) {
    const unsigned tid = threadIdx.x, lane = tid & 31u, lt = (1u << lane) - 1u;
    Ctr &C = S.ctr[w.ci];
    if (tid == 0) {
      S.kept = 0u;
      S.fmin = 0xFFFFFFFFu;
    }
    __syncthreads();
    unsigned lmin = 0xFFFFFFFFu;
    for (unsigned i0 = 0; i0 < w.F; i0 += BLOCK * 2u) {
      uint2 x[2];
      bool in[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const unsigned i = i0 + u * BLOCK + tid;
        in[u] = i < w.F;
        x[u] = in[u] ? __ldcg(w.L.far + i) : make_uint2(0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (in[u] && __ldcg(w.dist + x[u].x) != x[u].y) {
          in[u] = false;
          ++w.nstale;
        }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const bool nr = x[u].y < w.T;
        const unsigned bn = __ballot_sync(0xFFFFFFFFu, in[u] && nr);
        const unsigned bf = __ballot_sync(0xFFFFFFFFu, in[u] && !nr);
        if ((bn | bf) == 0u) continue;
        unsigned at = 0;
        if (lane < 2u) at = atomicAdd(lane ? &S.kept : &C.near_cnt, (unsigned)__popc(lane ? bf : bn));
        const unsigned pn = __shfl_sync(0xFFFFFFFFu, at, 0), pf = __shfl_sync(0xFFFFFFFFu, at, 1);
        if (pn + __popc(bn) > NS + w.L.ncap) C.stop = WV_ERR_OVERFLOW;
        if ((bn >> lane) & 1u) put(S, w, w.cur, pn + __popc(bn & lt), x[u]);
        if ((bf >> lane) & 1u) {
          __stcg(w.L.far + pf + __popc(bf & lt), x[u]);
          lmin = min(lmin, x[u].y);
        }
      }
    }
    lmin = __reduce_min_sync(0xFFFFFFFFu, lmin);
    if (lane == 0 && lmin != 0xFFFFFFFFu) atomicMin(&S.fmin, lmin);
    __syncthreads();
    w.F = S.kept;
  }

  /* Group exchange: every CTA publishes its frontier and its counts, and
   * takes an equal, contiguous share of the whole frontier back as its own
   * (neighbouring vertices stay together, so the hops that follow seldom
   * improve a vertex of another CTA).  False when the launch must end. */
  static __device__ bool exchange(const WvParams &P, Smem &S, State &w, unsigned cnt,
                                  unsigned fmin, unsigned stop, unsigned &round,
                                  unsigned long long deadline) {
    const unsigned tid = threadIdx.x, lane = tid & 31u, G = P.gsize;
    const unsigned group = blockIdx.x / G, rank = blockIdx.x % G;
    const unsigned par = round & 1u, xcap = NS + w.L.ncap;
    /* areas are the same size for every CTA of a group */
    const size_t stride = 2ull * w.L.ncap + w.L.fcap + w.L.scap + 2ull * xcap;
    uint2 *const mine = w.L.set + w.L.scap + (size_t)par * xcap;
    for (unsigned i = tid; i < min(cnt, xcap); i += BLOCK) __stcg(mine + i, entry(S, w, i));
    __syncthreads();
    /* The CTA's note carries the round: it is the arrival too.  One warp reads
     * every CTA's note until all are of this round.  Notes and published
     * frontiers alternate between two areas, so a CTA that runs ahead does not
     * write over what a slower one still reads. */
    ulonglong2 *const notes =
        reinterpret_cast<ulonglong2 *>(P.grp) + ((size_t)group * 2u + par) * WV_MAX_GROUP;
    ++round;
    const unsigned tag = round << WV_NOTE_BITS; /* low bits: the error, WV_SETTLED */
    ulonglong2 *const more = reinterpret_cast<ulonglong2 *>(P.grp) +
                             (size_t)P.groups * 2u * WV_MAX_GROUP +
                             ((size_t)group * 2u + par) * 2u * WV_MAX_GROUP;
    if (tid < 32u) {
      if (lane == 0) {
        if (PULL && w.trow && w.H) {
          __stcg(more + 2u * rank, make_ulonglong2(S.heavy, S.into));
          __stcg(more + 2u * rank + 1u, make_ulonglong2(w.H, S.smin));
        }
        __threadfence(); /* what the CTA published, before its note */
        st_note(notes + rank, min(cnt, xcap), w.F, fmin, tag | stop | (w.H ? WV_SETTLED : 0u));
      }
      constexpr unsigned J = WV_MAX_GROUP / 32u;
      unsigned c[J], far = 0, fx = 0, fm = 0xFFFFFFFFu, st = 0, it = 0;
      bool late = false;
      for (;;) {
        far = fx = st = 0u;
        fm = 0xFFFFFFFFu;
        bool here = true;
#pragma unroll
        for (unsigned j = 0; j < J; ++j) {
          const unsigned r = j * 32u + lane;
          uint4 x = make_uint4(0u, 0u, 0xFFFFFFFFu, tag);
          if (r < G) x = ld_note(notes + r);
          here = here && (x.w >> WV_NOTE_BITS) == (tag >> WV_NOTE_BITS);
          c[j] = x.x;
          far += x.y;
          fx = max(fx, x.y);
          fm = min(fm, x.z);
          st = wv_worse(st, x.w);
        }
        if (__all_sync(0xFFFFFFFFu, here)) break;
        late = (++it & 255u) == 0u && gtimer() > deadline;
        if (__any_sync(0xFFFFFFFFu, late)) break;
      }
      late = __any_sync(0xFFFFFFFFu, late);
      __threadfence(); /* the notes, before what they announce */
      unsigned tot = 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (unsigned j = 0; j < J; ++j) {
          const unsigned y = __shfl_up_sync(0xFFFFFFFFu, c[j], o);
          if (lane >= (unsigned)o) c[j] += y;
        }
      }
#pragma unroll
      for (unsigned j = 0; j < J; ++j) {
        c[j] += tot;
        tot = __shfl_sync(0xFFFFFFFFu, c[j], 31);
        if (j * 32u + lane < G) S.pre[j * 32u + lane] = c[j];
      }
      far = __reduce_add_sync(0xFFFFFFFFu, far);
      fx = __reduce_max_sync(0xFFFFFFFFu, fx);
      fm = __reduce_min_sync(0xFFFFFFFFu, fm);
      st = __reduce_max_sync(0xFFFFFFFFu, st & (WV_SETTLED - 1u)) |
           __reduce_or_sync(0xFFFFFFFFu, st & WV_SETTLED);
      /* first CTA whose entries reach into this CTA's share */
      const unsigned shr = ((tot + G - 1u) / G + 7u) & ~7u, lo = min(rank * shr, tot);
      unsigned first = 0;
#pragma unroll
      for (unsigned j = 0; j < J; ++j)
        first += __popc(__ballot_sync(0xFFFFFFFFu, j * 32u + lane < G && c[j] <= lo));
      if (PULL && w.trow && (st & WV_SETTLED) && tot <= P.low) {
        unsigned long long hv = 0, in = 0;
        unsigned ns = 0, sm = 0xFFFFFFFFu;
        for (unsigned r = lane; r < G; r += 32u) {
          if (!(ld_note(notes + r).w & WV_SETTLED)) continue;
          const ulonglong2 a = __ldcg(more + 2u * r), b = __ldcg(more + 2u * r + 1u);
          hv += a.x;
          in += a.y;
          ns += (unsigned)b.x;
          sm = min(sm, (unsigned)b.y);
        }
        for (int o = 16; o > 0; o >>= 1) {
          hv += __shfl_down_sync(0xFFFFFFFFu, hv, o);
          in += __shfl_down_sync(0xFFFFFFFFu, in, o);
        }
        ns = __reduce_add_sync(0xFFFFFFFFu, ns);
        sm = __reduce_min_sync(0xFFFFFFFFu, sm);
        if (lane == 0) {
          S.t_heavy = hv;
          S.t_into = in;
          S.t_set = ns;
          S.t_smin = sm;
        }
      }
      if (lane == 0) {
        S.tot = Note{tot, far, fm, st};
        S.far_max = fx;
        S.r0 = min(first, G - 1u);
        S.q = late ? 1u : 0u;
        if (late) atomicCAS(&P.st->err, 0u, WV_ERR_TIMEOUT);
      }
    }
    __syncthreads();
    if (S.q != 0u) return false; /* the wait ran out */
    const unsigned tot = S.tot.near_cnt;
    const unsigned shr = ((tot + G - 1u) / G + 7u) & ~7u;
    unsigned lo = min(rank * shr, tot), hi = min(lo + shr, tot), step = 1u, r = S.r0;
    if (POOL) { /* dealt out one by one: a long row's pieces lie together */
      lo = rank;
      hi = rank + (tot > rank ? (tot - rank + G - 1u) / G : 0u);
      step = G;
      r = 0u;
    }
    const uint2 *const base = mine - rank * stride; /* CTA 0 of the group      */
    for (unsigned j = tid; j < hi - lo; j += BLOCK) {
      const unsigned i = lo + j * step; /* below tot = pre[G - 1] */
      if (POOL) {
        unsigned top = G - 1u;
        while (r < top) {
          const unsigned mid = (r + top) >> 1;
          if (S.pre[mid] <= i) r = mid + 1u; else top = mid;
        }
      } else {
        while (S.pre[r] <= i) ++r;
      }
      put(S, w, w.cur, j, __ldcg(base + r * stride + (i - (r ? S.pre[r - 1] : 0u))));
    }
    if (tid == 0) {
      S.ctr[w.ci] = Ctr{hi - lo};
      S.ctr[next3(w.ci)] = Ctr{};
      if (hi - lo > NS + w.L.ncap) S.ctr[w.ci].stop = WV_ERR_OVERFLOW;
    }
    __syncthreads();
    return true;
  }

  static __device__ void run(const WvParams &P, Smem &S) {
    const unsigned tid = threadIdx.x, lane = tid & 31u;
    const unsigned rank = GRP ? blockIdx.x % P.gsize : 0u;
    const unsigned group = GRP ? blockIdx.x / P.gsize : blockIdx.x;
    const WvArea A = P.area[blockIdx.x];
    const unsigned inf = FLT ? ADDS_INF_F32_BITSV : ADDS_INF_I32_BITS;
    const unsigned long long deadline = gtimer() + P.timeout_ns;
    unsigned long long s_items = 0, s_hops = 0, s_splits = 0;
    State w;
    w.L.over = reinterpret_cast<uint2 *>(P.ws) + A.off;
    w.L.far = w.L.over + 2ull * A.ncap;
    w.L.set = w.L.far + A.fcap;
    w.L.ncap = A.ncap;
    w.L.fcap = A.fcap;
    w.L.scap = A.scap;
    w.npush = w.nstale = 0u;
    w.nedge = 0ull;
    unsigned err0 = *reinterpret_cast<volatile unsigned *>(&P.st->err), round = 0;
    for (unsigned turn = 0;; ++turn) {
      /* a CTA's next query: its own first, then from the counter; a group's:
       * from its share of the order */
      if (tid == 0) {
        const unsigned i = GRP ? (P.qoff ? P.qoff[group] : 0u) + turn
                               : (turn == 0 ? group : atomicAdd(&P.st->next, 1u) + P.groups);
        S.q = i < (GRP && P.qoff ? P.qoff[group + 1u] : P.nq) ? P.order[i] : 0xFFFFFFFFu;
        S.ctr[0] = Ctr{rank != 0u ? 0u : 1u, 0u, err0};
        S.ctr[1] = S.ctr[2] = Ctr{};
      }
      __syncthreads();
      const unsigned q = S.q;
      if (q == 0xFFFFFFFFu) break;
      const WvQuery Q = P.qs[q];
      w.row = Q.row;
      w.edges = Q.edges;
      w.first = Q.first;
      w.piece = Q.piece;
      w.split = Q.split;
      w.trow = PULL ? Q.trow : nullptr;
      w.np = Q.np;
      w.dist = Q.dist;
      w.n = Q.n;
      const unsigned src = (P.single_src != 0xFFFFFFFFu && q == 0u) ? P.single_src : Q.src;
      if (GRP && !P.filled) { /* an exchange follows before the first hop */
        for (unsigned i = rank * BLOCK + tid; i < Q.n; i += P.gsize * BLOCK)
          __stcg(Q.dist + i, i == src ? 0u : inf);
      }
      if (!GRP && !P.filled) {
        if ((reinterpret_cast<unsigned long long>(Q.dist) & 15ull) == 0ull) {
          const unsigned n4 = Q.n >> 2;
          for (unsigned i = tid; i < n4; i += BLOCK)
            __stcg(reinterpret_cast<uint4 *>(Q.dist) + i, make_uint4(inf, inf, inf, inf));
          if (tid < (Q.n & 3u)) __stcg(Q.dist + (n4 << 2) + tid, inf);
        } else {
          for (unsigned i = tid; i < Q.n; i += BLOCK) __stcg(Q.dist + i, inf);
        }
        __syncthreads();
        if (tid == 0) __stcg(Q.dist + src, 0u);
      }
      if (tid == 0) {
        S.nb[0][0] = make_uint2(src, 0u);
        S.heavy = S.into = 0ull;
        S.smin = 0xFFFFFFFFu;
        S.gsize = P.gsize;
      }
      __syncthreads();
      float delta = Q.delta;
      w.T = raise_word<FLT>(0u, delta);
      w.cur = w.ci = w.F = w.H = 0u;
      unsigned fmin = 0xFFFFFFFFu, hops = 0, split_at = GRP ? round : 0u, stop = 0;
      if (!GRP) {
        for (;;) {
          const Ctr c = S.ctr[w.ci];
          w.F += c.far_new;
          unsigned cnt = c.near_cnt;
          stop = c.stop;
          if (stop != 0u) break;
          if (cnt <= P.low && w.F != 0u) {
            /* a frontier that ran low again within a few hops: a wider step */
            if (hops - split_at <= 4u) delta *= 1.5f;
            split_at = hops;
            w.T = raise_word<FLT>(cnt == 0u && fmin != 0xFFFFFFFFu && fmin > w.T ? fmin : w.T, delta);
            split(S, w);
            fmin = S.fmin;
            cnt = S.ctr[w.ci].near_cnt;
            stop = S.ctr[w.ci].stop;
            __syncthreads();
            if (tid == 0) S.ctr[w.ci].far_new = 0u; /* in w.F already */
            ++s_splits;
            if (stop != 0u) break;
            if (cnt == 0u) {
              __syncthreads();
              if (w.F == 0u) break;
              continue;
            }
          }
          if (cnt == 0u) break;
          if (cnt > P.high) delta *= 0.75f;
          s_items += cnt;
          hop(S, w, cnt);
          ++hops;
          if (tid == 0 && (hops & 1023u) == 0u && gtimer() > deadline)
            S.ctr[next3(w.ci)].stop = WV_ERR_TIMEOUT;
          __syncthreads();
          w.cur ^= 1u;
          w.ci = next3(w.ci);
        }
      } else {
        /* A split leaves what it admits with the CTA that held it.  Where one
         * CTA holds much more than the others (steps narrower than most
         * weights: nothing of the first hops is dealt out) its entries are
         * dealt out before they are relaxed (ER 300,000 x 16 with weights 1 to
         * 10 overflowed the first CTA's list). */
        bool deal = !P.filled;
        unsigned long long gone = 0; /* in-edges of settled vertices */
        for (;;) {
          /* up to P.hops hops on this CTA's own entries */
          const unsigned hmax = deal ? 0u : Q.hops;
          const bool dealt = deal;
          deal = false;
          unsigned cnt = 0;
          for (unsigned h = 0;; ++h) {
            const Ctr c = S.ctr[w.ci];
            w.F += c.far_new;
            w.H += c.set_new;
            cnt = c.near_cnt;
            stop = c.stop;
            if (h == hmax || cnt == 0u || stop != 0u || (h != 0u && (cnt > BLOCK / 2u || c.cut != 0u)))
              break;
            s_items += cnt;
            if (POOL) hop_pool(S, w, cnt); else hop(S, w, cnt);
            ++hops;
            __syncthreads();
            w.cur ^= 1u;
            w.ci = next3(w.ci);
          }
          if (!exchange(P, S, w, cnt, fmin, stop, round, deadline)) {
            stop = WV_ERR_TIMEOUT;
            break;
          }
          const Note t = S.tot;
          stop = t.stop & ~WV_SETTLED;
          const bool settled = (t.stop & WV_SETTLED) != 0u;
          if (stop != 0u || (t.near_cnt == 0u && t.far_cnt == 0u && !settled)) break;
          const bool few = t.near_cnt <= P.low && !(dealt && t.near_cnt != 0u);
          if (POOL && few && settled) {
            bool pulled = false;
            if constexpr (PULL) if (w.trow) {
              /* in-edges of the vertices that have not settled yet: a pull reads
               * at most these */
              gone += S.t_into;
              const unsigned long long left = Q.m > gone ? Q.m - gone : 0ull;
              if (S.t_set > Q.n >> 6 && S.t_heavy > left) {
                unsigned ne = 0;
                w.npush += pull(S, w, Q.tedges, add_word<FLT>(S.t_smin, Q.thr), ne);
                w.nedge += ne;
                w.H = 0u;
                pulled = deal = true;
              }
              __syncthreads(); /* totals and sums are read */
              if (tid == 0) {
                S.heavy = S.into = 0ull;
                S.smin = 0xFFFFFFFFu;
              }
            }
            if (!pulled) unsettle(S, w);
          } else if (few && t.far_cnt != 0u) {
            deal = S.far_max > 256u && (unsigned long long)S.far_max * P.gsize * 2u > 3ull * t.far_cnt;
            if (Q.grow && round - split_at <= 1u) delta *= 1.5f;
            split_at = round;
            w.T = raise_word<FLT>(
                t.near_cnt == 0u && t.far_min != 0xFFFFFFFFu && t.far_min > w.T ? t.far_min : w.T, delta);
            split(S, w);
            fmin = S.fmin;
            ++s_splits;
          } else if (Q.grow && t.near_cnt > P.high) {
            delta *= 0.75f;
          }
          __syncthreads();
          if (gtimer() > deadline && tid == 0 && rank == 0u) S.ctr[w.ci].stop = WV_ERR_TIMEOUT;
          __syncthreads();
        }
      }
      s_hops += hops;
      if (stop != 0u && tid == 0) atomicCAS(&P.st->err, 0u, stop);
      __syncthreads(); /* S is read to the end before the next query's setup */
      if (stop != 0u) break;
    }
    unsigned long long s_edge = w.nedge, s_push = w.npush, s_stale = w.nstale;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s_edge += __shfl_down_sync(0xFFFFFFFFu, s_edge, o);
      s_push += __shfl_down_sync(0xFFFFFFFFu, s_push, o);
      s_stale += __shfl_down_sync(0xFFFFFFFFu, s_stale, o);
    }
    if (lane == 0) {
      if (s_edge) atomicAdd(&P.st->edges, s_edge);
      if (s_push) atomicAdd(&P.st->pushes, s_push);
      if (s_stale) atomicAdd(&P.st->stale, s_stale);
      if (tid == 0) {
        atomicAdd(&P.st->items, s_items);
        if (rank == 0u) {
          atomicAdd(&P.st->steps, GRP ? (unsigned long long)round : s_hops);
          atomicAdd(&P.st->splits, s_splits);
        }
      }
    }
  }
};

template <bool FLT, int BLOCK, int NS, int MINB, bool GRP, int PL>
__global__ void __launch_bounds__(BLOCK, MINB) wave_kernel(const __grid_constant__ WvParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Wave<FLT, BLOCK, NS, GRP, PL>::run(P, *reinterpret_cast<WSmem<BLOCK, NS, PL> *>(smem_raw));
}

/* INF everywhere and 0 at the source, by the whole GPU */
__global__ void wave_fill(const WvQuery *qs, unsigned single_src, unsigned inf) {
  const WvQuery Q = qs[0];
  const unsigned src = single_src != 0xFFFFFFFFu ? single_src : Q.src;
  for (unsigned v = blockIdx.x * blockDim.x + threadIdx.x; v < Q.n; v += gridDim.x * blockDim.x)
    Q.dist[v] = v == src ? 0u : inf;
}

template <bool FLT, int BLOCK, int NS, int MINB, bool GRP, int PL>
static cudaError_t resident(int *bps) {
  const int smem = (int)sizeof(WSmem<BLOCK, NS, PL>);
  auto *k = wave_kernel<FLT, BLOCK, NS, MINB, GRP, PL>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k, BLOCK, smem);
}

template <bool FLT, int BLOCK, int NS, int MINB, bool GRP, int PL>
static cudaError_t launch(const WvParams &P, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.groups * P.gsize);
  cfg.blockDim = dim3(BLOCK);
  cfg.dynamicSmemBytes = sizeof(WSmem<BLOCK, NS, PL>);
  cfg.stream = st;
  /* the CTAs of a group wait for each other: all must be resident */
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = GRP ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, wave_kernel<FLT, BLOCK, NS, MINB, GRP, PL>, P);
}

}  // namespace adds_wave

/* (variant, threads, frontier entries in shared memory, CTAs per SM the
 * registers are sized for, several CTAs per query, pooled edges and pulls, entries per
 * CTA below which a frontier takes more of the far list).  The batch of 128
 * grids x 16 sources: 256 threads x 4 7.2 ms, x 5 7.6, x 6 8.2, 128 x 10 11.4,
 * 512 x 3 7.8, 1024 x 1 14.5.  Low marks: 32 entries 7.6 ms, 16 7.7, 64 8.0, 0
 * 8.2 there; 4096^2 grid on 148 CTAs 2,500 entries 18.3 ms, 1,000 19.3, 9,500
 * 21.7. */
#define WV_SHAPES(X)                           \
  X(WV_CTA, 256, 1024, 4, false, 0, 32)        \
  X(WV_WIDE, 1024, 4096, 1, false, 0, 64)      \
  X(WV_GROUP, 512, 2048, 1, true, 0, 16)       \
  X(WV_POOL, 1024, 2048, 1, true, 1, 8)        \
  X(WV_PULL, 1024, 2048, 1, true, 2, 8)

static unsigned wv_block(int shape) {
#define X(s, b, ns, m, g, pl, lo) if (shape == s) return b;
  WV_SHAPES(X)
#undef X
  return 0;
}
static unsigned wv_low(int shape) {
#define X(s, b, ns, m, g, pl, lo) if (shape == s) return lo;
  WV_SHAPES(X)
#undef X
  return 0;
}
unsigned wv_near(int shape) {
#define X(s, b, ns, m, g, pl, lo) if (shape == s) return ns;
  WV_SHAPES(X)
#undef X
  return 0;
}

void wv_engine_free(WvEngine &E) {
  void *ptrs[] = {E.qs, E.order, E.area, E.ws, E.st, E.grp};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (E.st_host) cudaFreeHost(E.st_host);
  E = WvEngine();
}

int wv_engine_reset(WvEngine &E, cudaStream_t st) {
  return cudaMemsetAsync(E.st, 0, sizeof(WvStat), st) == cudaSuccess &&
                 cudaStreamSynchronize(st) == cudaSuccess
             ? 0
             : -5;
}

int wv_engine_upload(WvEngine &E, cudaStream_t st) {
  return cudaMemcpyAsync(E.qs, E.qs_host.data(), E.qs_host.size() * sizeof(WvQuery),
                         cudaMemcpyHostToDevice, st) == cudaSuccess &&
                 cudaStreamSynchronize(st) == cudaSuccess
             ? 0
             : -5;
}

static int engine_layout(WvEngine &E, int device, bool flt, int shape, unsigned gsize,
                         const std::vector<WvQuery> &qv, cudaStream_t st) {
  using namespace adds_wave;
  E.device = device;
  E.flt = flt;
  E.shape = shape;
  E.nq = (unsigned)qv.size();
  E.qs_host = qv;
  int sms = 0, bps = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return -5;
  E.kernel = shape;
  for (const WvQuery &q : qv)
    if (shape == WV_POOL && q.trow) E.kernel = WV_PULL;
  const cudaError_t e = wv_prepare(flt, E.kernel, &bps);
  if (e != cudaSuccess || bps < 1) {
    cudaGetLastError();
    return -9;
  }
  const bool grp = shape == WV_GROUP || shape == WV_POOL;
  for (WvQuery &q : E.qs_host) wv_query_schedule(q, shape);
  E.gsize = grp ? std::min(gsize ? gsize : (unsigned)sms, std::min((unsigned)sms, (unsigned)WV_MAX_GROUP)) : 1u;
  E.req_gsize = gsize;
  E.has_set = false;
  for (const WvQuery &q : qv) E.has_set = E.has_set || (shape == WV_POOL && q.split);
  E.groups = grp ? std::min((unsigned)sms / E.gsize, E.nq) : std::min((unsigned)(bps * sms), E.nq);
  E.ctas = E.groups * E.gsize;
  /* largest first: the last group to finish is not stuck with a big query */
  std::vector<unsigned> order(E.nq);
  for (unsigned i = 0; i < E.nq; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](unsigned a, unsigned b) {
    return qv[a].m + qv[a].n > qv[b].m + qv[b].n;
  });
  /* Several groups: each its own share of the queries, the next largest one to
   * the group with the least to do so far (edges, and the hops of any query
   * as 500,000 edges a CTA). */
  std::vector<unsigned> qoff;
  if (grp && E.nq > 1u) {
    std::vector<std::vector<unsigned>> share(E.groups);
    std::vector<double> load(E.groups, 0.0);
    for (unsigned i : order) {
      const size_t g = std::min_element(load.begin(), load.end()) - load.begin();
      share[g].push_back(i);
      load[g] += (double)qv[i].m + 5e5 * E.gsize;
    }
    order.clear();
    for (const auto &v : share) {
      qoff.push_back((unsigned)order.size());
      order.insert(order.end(), v.begin(), v.end());
    }
    qoff.push_back((unsigned)order.size());
  }
  /* A CTA's lists hold the queries it may meet: its own first one and any
   * later one.  A road's wave front is a small part of its graph: frontier
   * n/4 (and the shared entries) and far list n/2 in all.  A graph with longer
   * rows has most of its vertices pending at once, some of them several times.
   * Either way one CTA may hold much more than its share for a few hops.
   * Where that is not enough, the launch reports an overflow. */
  bool dense = false;
  for (const WvQuery &q : qv) dense = dense || q.m >= 6ull * q.n;
  std::vector<WvArea> area;
  std::vector<unsigned> maxn(E.nq);
  for (unsigned i = E.nq, mx = 0; i-- > 0;) {
    mx = std::max(mx, qv[order[i]].n);
    maxn[i] = mx;
  }
  if (!qoff.empty()) /* a group meets its own share only, the largest first */
    for (unsigned g = 0; g < E.groups; ++g) {
      maxn[g] = 0;
      for (unsigned i = qoff[g]; i < qoff[g + 1]; ++i) maxn[g] = std::max(maxn[g], qv[order[i]].n);
    }
  unsigned long long tot = 0;
  for (;;) {
    area.clear();
    tot = 0;
    for (unsigned g = 0; g < E.groups; ++g)
      for (unsigned r = 0; r < E.gsize; ++r) {
        const unsigned long long n = maxn[g], cl = E.gsize;
        WvArea A;
        A.off = tot;
        /* (side by side, half of that: the lists of a group of two CTAs on a
         * graph of 10^6 vertices take 50 MB) */
        A.fcap = (unsigned)((dense ? (E.groups > 1u ? 2u : 4u) * n : n / 2u) / cl +
                            std::min(dense ? 2ull * n : n, dense ? 65536ull : 32768ull));
        /* a group's CTA may find its whole far list below a raised threshold */
        A.ncap = grp ? (E.groups > 1u ? A.fcap / 2u : A.fcap) : (unsigned)((dense ? n : n / 4u) + std::min(n, 16384ull));
        tot += 2ull * A.ncap + A.fcap;
        A.scap = E.has_set ? (unsigned)((E.groups > 1u ? 1u : 2u) * n / cl + std::min(n, 32768ull)) : 0u;
        tot += A.scap;
        if (grp) tot += 2ull * (wv_near(shape) + A.ncap); /* published frontiers */
        area.push_back(A);
      }
    /* at most 8 GB of lists: fewer queries side by side, if need be */
    if (tot <= (1ull << 30)) break;
    if (grp || E.groups <= 8u) return -4;
    E.groups /= 2u;
  }
  E.ctas = E.groups * E.gsize;
#define WV_ALLOC(ptr, bytes_)                             \
  do {                                                    \
    const size_t _b = (bytes_);                           \
    if (cudaMalloc((void **)&(ptr), _b) != cudaSuccess) { \
      cudaGetLastError();                                 \
      return -4;                                          \
    }                                                     \
    E.bytes += _b;                                        \
  } while (0)
  WV_ALLOC(E.qs, (size_t)E.nq * sizeof(WvQuery));
  WV_ALLOC(E.order, (size_t)(E.nq + E.groups + 1u) * 4);
  WV_ALLOC(E.area, (size_t)E.ctas * sizeof(WvArea));
  WV_ALLOC(E.ws, (size_t)tot * 8);
  WV_ALLOC(E.st, sizeof(WvStat));
  WV_ALLOC(E.grp, (size_t)E.groups * WV_GRP_WORDS * 4);
#undef WV_ALLOC
  if (cudaMallocHost((void **)&E.st_host, sizeof(WvStat)) != cudaSuccess) {
    cudaGetLastError();
    return -4;
  }
  memset(E.st_host, 0, sizeof(WvStat));
  E.shares = !qoff.empty();
  order.insert(order.end(), qoff.begin(), qoff.end());
  if (cudaMemcpyAsync(E.order, order.data(), order.size() * 4, cudaMemcpyHostToDevice, st) !=
          cudaSuccess ||
      cudaMemcpyAsync(E.area, area.data(), area.size() * sizeof(WvArea), cudaMemcpyHostToDevice,
                      st) != cudaSuccess)
    return -5;
  const int rc = wv_engine_upload(E, st);
  return rc ? rc : wv_engine_reset(E, st);
}

/* gsize: CTAs per query of the group variants (0: one per SM).  E is whole
 * afterwards or, on an error, empty: callers take an engine of the right
 * variant and number of queries to be ready for use. */
int wv_engine_alloc(WvEngine &E, int device, bool flt, int shape, unsigned gsize,
                    const std::vector<WvQuery> &qv, cudaStream_t st) {
  wv_engine_free(E);
  const int rc = engine_layout(E, device, flt, shape, gsize, qv, st);
  if (rc) wv_engine_free(E);
  return rc;
}

void wv_schedule(WvParams &P, int shape) {
  P.low = wv_low(shape) * P.gsize;
  P.high = wv_block(shape) * P.gsize * 4u;
}

void wv_query_schedule(WvQuery &q, int shape) {
  /* Hops on a CTA's own entries between two exchanges.  Roads: 8 (a 4096^2
   * grid 18.3 ms, against 19.3 at 4 and 33 at 1, where the exchanges cost more
   * than the hops).  Pooled: 1, since the neighbours of an entry are anywhere
   * and hops on stale distances relax too much (R-MAT 16 0.38 ms, 0.60 at 8),
   * but 8 on graphs so small that the few hops are all there is (20,000
   * vertices 0.20 ms, 0.27 at 1). */
  q.hops = shape == WV_GROUP || (q.n < 32768u && !q.piece) ? 8u : 1u;
  /* a pooled frontier widens its step only on small graphs, whose few hops are
   * all latency: elsewhere a wide step relaxes rows again and again (ER 10^6 x 8
   * 3.1 edges relaxed per edge and 0.90 ms with, 1.1 and 0.69 without; R-MAT 16
   * 0.38 ms with, 0.42 without) */
  q.grow = shape != WV_POOL || q.n < (1u << 17) ? 1u : 0u;
}

cudaError_t wv_prepare(bool flt, int shape, int *bps) {
  using namespace adds_wave;
#define X(s, b, ns, m, g, pl, lo) \
  if (shape == s)                 \
    return flt ? resident<true, b, ns, m, g, pl>(bps) : resident<false, b, ns, m, g, pl>(bps);
  WV_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

cudaError_t wv_launch(const WvParams &P, bool flt, int shape, cudaStream_t st) {
  using namespace adds_wave;
#define X(s, b, ns, m, g, pl, lo) \
  if (shape == s)                 \
    return flt ? launch<true, b, ns, m, g, pl>(P, st) : launch<false, b, ns, m, g, pl>(P, st);
  WV_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

int wv_engine_enqueue(WvEngine &E, unsigned single_src, unsigned long long timeout_ns,
                      cudaStream_t st, cudaEvent_t k0, cudaEvent_t k1) {
  using namespace adds_wave;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) return -5;
  const unsigned fl = cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : 0u;
  const size_t keep = offsetof(WvStat, next); /* the error word stays */
  if (cudaMemsetAsync(reinterpret_cast<char *>(E.st) + keep, 0, sizeof(WvStat) - keep, st) !=
      cudaSuccess)
    return -5;
  WvParams P;
  memset(&P, 0, sizeof P);
  P.qs = E.qs;
  P.order = E.order;
  P.qoff = E.shares ? E.order + E.nq : nullptr;
  P.nq = E.nq;
  P.groups = E.groups;
  P.gsize = E.gsize;
  P.area = E.area;
  P.ws = E.ws;
  P.st = E.st;
  P.grp = E.grp;
  P.single_src = single_src;
  P.timeout_ns = timeout_ns;
  wv_schedule(P, E.shape);
  const bool grp = E.shape == WV_GROUP || E.shape == WV_POOL;
  P.filled = E.nq == 1u && (grp || E.qs_host[0].n > (1u << 18)) ? 1u : 0u;
  E.fills = P.filled != 0u;
  if (grp && cudaMemsetAsync(E.grp, 0, (size_t)E.groups * 2u * 16u * WV_MAX_GROUP, st) != cudaSuccess) return -5;
  if (P.filled)
    wave_fill<<<1184, 256, 0, st>>>(E.qs, single_src,
                                    E.flt ? ADDS_INF_F32_BITSV : ADDS_INF_I32_BITS);
  if (k0 && cudaEventRecordWithFlags(k0, st, fl) != cudaSuccess) return -5;
  if (wv_launch(P, E.flt, E.kernel, st) != cudaSuccess) return -5;
  if (k1 && cudaEventRecordWithFlags(k1, st, fl) != cudaSuccess) return -5;
  if (cudaMemcpyAsync(E.st_host, E.st, sizeof(WvStat), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return -5;
  return 0;
}

int wv_engine_status(const WvEngine &E, char *msg, size_t msg_len) {
  const unsigned err = E.st_host->err;
  if (err && msg) snprintf(msg, msg_len, "wave kernel: device error %u", err);
  return err == 0u ? 0 : (err == WV_ERR_OVERFLOW ? -7 : -6);
}
