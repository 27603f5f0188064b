/*
 * adjoint.cu — dL/dw of batched SSSP distances (float graphs).
 *
 * No reference counterpart: the reference only computes distances.  With
 * d(t) = fold of fl(d + w) along the shortest path, the (sub)gradient taken
 * along the shortest-path tree is dd(t)/dw_e = 1 if e lies on the tree path
 * to t.  So with lambda[v] = dL/dd[v] + sum over tree children c of
 * lambda[c], dL/dw_pred(v) = lambda[v].
 *
 * Determinism:
 *   - pred(v) = the tight in-edge e=(u->v), fl(d[u]+w_e) == d[v] with
 *     d[u] < d[v], of smallest CSR index (64-bit atomicMin on e<<32|u);
 *     vertices reached only through zero-gap tight edges (d[u] == d[v])
 *     get their parent in breadth-first rounds from already-treed vertices,
 *     again smallest index first, so the tree never has a cycle;
 *   - lambda[x] = seed[x] + lambda of x's children summed in x's CSR edge
 *     order, computed by the last child to finish ("last arriver
 *     continues" up the tree): no float atomics, fixed summation order;
 *   - grad[e] sums the queries of a graph in query order.
 * The CPU oracle's adjoint (oracle_adjoint in oracle/oracle.c) follows the
 * same orders, so the gradient is bit-exact against it.
 */
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "../../include/adds.h"
#include "adds_internal.h"

struct adds_graph;
struct adds_batch;
int adds_batch_internal(adds_batch *b, cudaStream_t *st, unsigned *nq,
                        std::vector<adds_graph *> **qgraph, std::vector<uint32_t> **srcs,
                        std::vector<adds_graph *> **ugraph, std::vector<unsigned> **qgid,
                        unsigned **dist_all, std::vector<size_t> **dist_off, void ***adj);
void adds_graph_internal(const adds_graph *g, const unsigned **row, const uint2 **edges,
                         uint32_t *n, uint64_t *m, unsigned *max_deg, int *device);

#define NO_PRED 0xFFFFFFFFFFFFFFFFull
#define NO_ROUND 0xFFFFFFFFu

struct AdjQ {
  const unsigned *row;
  const uint2 *edges;
  const float *dist;
  const float *seed; /* dL/d dist */
  unsigned long long *pred;
  unsigned long long *lam; /* low half: lambda once it is known; until then
                              what the children leave for each other       */
  unsigned *kids; /* rows of at most 32 edges: which of them are tree edges;
                     longer rows in the launch: how many are               */
  unsigned *round;
  unsigned n;
  unsigned src;
  unsigned tile0; /* first tile of the query (TILE vertices each)          */
};

struct AdjG { /* one distinct graph and the queries that use it */
  const uint2 *edges;
  float *grad;
  unsigned m;
  unsigned q_begin, q_end; /* into the query-index list */
  unsigned tile0;          /* first tile of the graph (TILE edges each)    */
};

namespace adj {

constexpr unsigned TILE = 4096; /* vertices (or edges) a CTA takes            */

/* The query (or graph) a CTA's tile belongs to and its first vertex (edge).
 * One CTA per tile: a grid as long as the largest query for every query of a
 * batch would be mostly empty CTAs (128 grids of side 64 to 512: 0.9 ms a
 * kernel, whatever it did). */
template <class T>
__device__ __forceinline__ unsigned locate(const T *a, unsigned cnt, unsigned &first) {
  unsigned lo = 0, hi = cnt - 1u;
  while (lo < hi) {
    const unsigned mid = (lo + hi + 1u) >> 1;
    if (a[mid].tile0 <= blockIdx.x) lo = mid; else hi = mid - 1u;
  }
  first = (blockIdx.x - a[lo].tile0) * TILE;
  return lo;
}
#define ADJ_TILE(q, v0, v1)                               \
  unsigned v0;                                            \
  const AdjQ &q = qs[locate(qs, nq, v0)];                 \
  const unsigned v1 = min(q.n, v0 + TILE);

__global__ void k_init(const AdjQ *qs, unsigned nq) {
  ADJ_TILE(q, v0, v1)
  for (unsigned v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
    q.pred[v] = NO_PRED;
    q.lam[v] = 0ull;
    q.kids[v] = 0u;
  }
}

/* strict tight edges: d[u] < d[v] and fl(d[u] + w) == d[v].  Unreached vertices
 * have none, although a weight near FLT_MAX can round to their distance word:
 * no walk starts at them, and a parent would wait for one. */
__global__ void k_pred_strict(const AdjQ *qs, unsigned nq) {
  ADJ_TILE(q, v0, v1)
  for (unsigned u = v0 + threadIdx.x; u < v1; u += blockDim.x) {
    const float du = q.dist[u];
    if (__float_as_uint(du) == ADDS_INF_F32_BITSV) continue;
    const unsigned e1 = q.row[u + 1];
    for (unsigned e = q.row[u]; e < e1; ++e) {
      const uint2 ed = q.edges[e];
      if (ed.x == q.src) continue;
      const float dv = q.dist[ed.x];
      if (du < dv && __float_as_uint(dv) != ADDS_INF_F32_BITSV &&
          __fadd_rn(du, __uint_as_float(ed.y)) == dv)
        atomicMin(&q.pred[ed.x], ((unsigned long long)e << 32) | u);
    }
  }
}

/* Marks each vertex at its parent (MASK: the bit of its tree edge in the
 * parent's row; else a count), and counts the reached vertices left without a
 * parent. */
template <bool MASK>
__global__ void k_children(const AdjQ *qs, unsigned nq, unsigned *orphans) {
  ADJ_TILE(q, v0, v1)
  unsigned c = 0;
  for (unsigned v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
    const unsigned long long p = q.pred[v];
    if (p != NO_PRED) {
      const unsigned u = (unsigned)p;
      if (MASK) atomicOr(&q.kids[u], 1u << ((unsigned)(p >> 32) - q.row[u]));
      else atomicAdd(&q.kids[u], 1u);
    } else if (v != q.src && __float_as_uint(q.dist[v]) != ADDS_INF_F32_BITSV) {
      ++c;
    }
  }
  if (c) atomicAdd(orphans, c);
}

/* Zero-gap ties only: rounds start from the vertices that have a parent, and
 * the children are counted again afterwards. */
__global__ void k_rounds_init(const AdjQ *qs, unsigned nq) {
  ADJ_TILE(q, v0, v1)
  for (unsigned v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
    q.round[v] = (v == q.src || q.pred[v] != NO_PRED) ? 0u : NO_ROUND;
    q.kids[v] = 0u;
  }
}

/* breadth-first round r over zero-gap tight edges */
__global__ void k_pred_zero(const AdjQ *qs, unsigned nq, unsigned r, unsigned *changed) {
  ADJ_TILE(q, v0, v1)
  for (unsigned u = v0 + threadIdx.x; u < v1; u += blockDim.x) {
    if (q.round[u] >= r) continue; /* u must be in the tree before round r */
    const float du = q.dist[u];
    const unsigned e1 = q.row[u + 1];
    for (unsigned e = q.row[u]; e < e1; ++e) {
      const uint2 ed = q.edges[e];
      if (ed.x == q.src) continue;
      if (q.round[ed.x] < r) continue; /* already in the tree */
      const float dv = q.dist[ed.x];
      if (du == dv && __fadd_rn(du, __uint_as_float(ed.y)) == dv) {
        atomicMin(&q.pred[ed.x], ((unsigned long long)e << 32) | u);
        atomicMin(&q.round[ed.x], r);
        *changed = 1u;
      }
    }
  }
}

__device__ __forceinline__ float lam_of(const AdjQ &q, unsigned v) {
  return __uint_as_float((unsigned)__ldcg(q.lam + v));
}

/* acc (the seed of x) plus lambda of x's children, in x's CSR edge order */
template <bool MASK>
__device__ __forceinline__ float gather_lambda(const AdjQ &q, unsigned x, unsigned kids, float acc) {
  const unsigned r0 = __ldg(q.row + x);
  if (MASK) {
    for (; kids; kids &= kids - 1u)
      acc = __fadd_rn(acc, lam_of(q, __ldg(&q.edges[r0 + (unsigned)__ffs(kids) - 1u].x)));
    return acc;
  }
  const unsigned e1 = __ldg(q.row + x + 1);
  for (unsigned e = r0; e < e1; ++e) {
    const unsigned v = q.edges[e].x;
    const unsigned long long p = __ldg(&q.pred[v]);
    if ((unsigned)(p >> 32) == e && p != NO_PRED) acc = __fadd_rn(acc, lam_of(q, v));
  }
  return acc;
}

/* A walk handed from the first launch of walks to the second. */
struct __align__(16) Walk {
  unsigned q, x;
  float acc; /* lambda of x, complete */
  unsigned pad;
};

/* Every leaf of the tree starts a walk to the root; the last child of a vertex
 * to finish carries on with it.  An only child carries on without asking; of
 * two, the first leaves its lambda in the parent's word and the second takes
 * it with the same exchange; of more, each counts itself there and the last
 * reads the others'.  So a step is one round trip for what the parent needs and
 * mostly at most one atomic, with no fence; lanes that do need fences wait until
 * SLOW of the warp do, since the others would wait with them.
 *
 * Bound by those round trips and by the lanes that take part: walks are a few
 * steps long on average and hundreds at worst.  FIRST: a warp takes the leaves
 * of neighbouring vertices, a lane whose walk has ended takes the next leaf,
 * and once the leaves are out and at most HAND walks go on these are handed to
 * a second launch: long walks would keep a CTA's place on the SM for a lane or
 * two (a third of the warps resident, 17 lanes active).  That launch gives each
 * warp HAND walks at a time.
 * 128 grids x 16 sources: 37 ms when the lanes of a warp waited for the longest
 * of their 32 walks; 15 with lanes refilled but a fence, a count and a read of
 * every child at each vertex; 9.0 with exchanges instead; 3.8 + 3.1 now. */
constexpr unsigned SLOW = 8u, HAND = 4u;
template <bool MASK, bool FIRST, bool HANDS>
__global__ void __launch_bounds__(512, 2) k_walk(const AdjQ *qs, unsigned nq, Walk *hand,
                                                 unsigned *ctr) {
  /* ctr: walks handed over, walks taken up */
  const unsigned lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  __shared__ unsigned short list[FIRST ? TILE : 1u];
  unsigned t0 = 0, qi = 0, end = 0, next = 0, v0 = 0;
  const unsigned own = TILE / (blockDim.x / 32u), at = FIRST ? (threadIdx.x >> 5) * own : 0u;
  unsigned short *const leaf = list + at;
  if (FIRST) qi = locate(qs, nq, t0);
  AdjQ q = qs[qi];
  if (FIRST) { /* the leaves among the warp's vertices */
    v0 = t0 + at;
    const unsigned v1 = min(q.n, v0 + own);
#pragma unroll 4
    for (unsigned i = v0; i < v1; i += 32u) {
      const unsigned v = i + lane;
      const bool is = v < v1 && __ldg(q.kids + v) == 0u &&
                      __float_as_uint(__ldg(q.dist + v)) != ADDS_INF_F32_BITSV;
      const unsigned b = __ballot_sync(0xFFFFFFFFu, is);
      if (is) leaf[end + __popc(b & lt)] = (unsigned short)(v - v0);
      end += __popc(b);
    }
    __syncwarp();
  } else {
    end = ctr[0];
  }
  bool busy = false;
  unsigned x = 0;
  float acc = 0.f;                /* lambda of x, complete */
  unsigned long long p = NO_PRED; /* pred of x */
  unsigned kids = 0, k = 0;       /* children of x (k: 1, 2 or more)            */
  float seed = 0.f;
  while (next < end || __any_sync(0xFFFFFFFFu, busy)) {
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, !busy);
    bool fresh = false; /* its first loads overlap the other lanes' step */
    if (FIRST) { /* idle lanes take the next leaves */
      const unsigned i = next + __popc(idle & lt);
      if (!busy && i < end) {
        busy = fresh = true;
        x = v0 + leaf[i];
        k = 0u;
        acc = q.seed ? __ldg(q.seed + x) : 0.f;
        p = __ldg(&q.pred[x]);
      }
      next += __popc(idle);
    } else if (next < end && (idle & ((1u << HAND) - 1u))) { /* or the next walks */
      unsigned i = end;
      if (!busy && lane < HAND) i = atomicAdd(ctr + 1, 1u);
      if (i < end) {
        const Walk w = hand[i];
        busy = fresh = true;
        q = qs[w.q];
        x = w.x;
        k = 0u;
        acc = w.acc;
        p = __ldg(&q.pred[x]);
      }
      /* the counter only rises: once past the end nothing is left */
      if (__any_sync(0xFFFFFFFFu, !busy && lane < HAND)) next = end;
    }
    if (busy && !fresh && k <= 2u) {
      __stcg(reinterpret_cast<unsigned *>(q.lam + x), __float_as_uint(acc));
      busy = p != NO_PRED; /* else the source (or an unreached root) */
      if (busy) {
        const unsigned e = (unsigned)(p >> 32);
        x = (unsigned)p; /* the parent; acc is its child's until it is complete */
        kids = __ldg(q.kids + x);
        const unsigned r0 = MASK ? __ldg(q.row + x) : 0u;
        seed = q.seed ? __ldg(q.seed + x) : 0.f;
        p = __ldg(&q.pred[x]);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(q.lam + x));
        k = MASK ? (unsigned)__popc(kids) : kids;
        if (k == 1u) {
          acc = __fadd_rn(seed, acc);
        } else if (MASK && k == 2u) {
          const unsigned long long old =
              atomicExch(q.lam + x, (1ull << 32) | __float_as_uint(acc));
          busy = (old >> 32) != 0ull; /* else the sibling still runs */
          const float other = __uint_as_float((unsigned)old);
          const bool mine = (kids & (0u - kids)) == 1u << (e - r0); /* this child's edge first */
          acc = __fadd_rn(__fadd_rn(seed, mine ? acc : other), mine ? other : acc);
        } else {
          k = 3u; /* waits for the slow way below */
        }
      }
    }
    const unsigned slow = __ballot_sync(0xFFFFFFFFu, busy && k > 2u);
    const unsigned going = __ballot_sync(0xFFFFFFFFu, busy);
    const bool last = HANDS && next >= end && __popc(going) <= (int)HAND;
    if (slow != 0u && (last || __popc(slow) >= (int)(FIRST ? SLOW : 1u) || slow == going)) {
      if (busy && k > 2u) {
        const unsigned all = MASK ? (unsigned)__popc(kids) : kids;
        /* lambda of the child, before it counts as finished; the siblings'
         * counts, before their lambdas are read */
        unsigned long long old;
        asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;"
                     : "=l"(old) : "l"(q.lam + x), "l"(1ull << 32) : "memory");
        busy = (unsigned)(old >> 32) + 1u == all; /* else siblings still run */
        if (busy) acc = gather_lambda<MASK>(q, x, kids, seed);
        k = 1u;
      }
    }
    if (last) {
      const unsigned b = __ballot_sync(0xFFFFFFFFu, busy);
      unsigned i = 0;
      if (lane == 0 && b) i = atomicAdd(ctr, (unsigned)__popc(b));
      i = __shfl_sync(0xFFFFFFFFu, i, 0);
      if (busy) hand[i + __popc(b & lt)] = Walk{qi, x, acc, 0u};
      break;
    }
  }
}

/* grad[e] (+)= sum over the graph's queries, in query order, of lambda at
 * dst(e) when e is that vertex's tree edge */
__global__ void k_grad(const AdjG *gs, unsigned ng, const AdjQ *qs, const unsigned *qidx,
                       int accumulate) {
  unsigned e0;
  const AdjG &g = gs[locate(gs, ng, e0)];
  const unsigned e1 = (unsigned)min((unsigned long long)g.m, (unsigned long long)e0 + TILE);
  for (unsigned e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const unsigned v = g.edges[e].x;
    float acc = 0.f;
    for (unsigned i = g.q_begin; i < g.q_end; ++i) {
      const AdjQ &q = qs[qidx[i]];
      const unsigned long long p = q.pred[v];
      if (p != NO_PRED && (unsigned)(p >> 32) == e) acc = __fadd_rn(acc, __uint_as_float((unsigned)q.lam[v]));
    }
    g.grad[e] = accumulate ? __fadd_rn(g.grad[e], acc) : acc;
  }
}

}  // namespace adj

/* scratch kept with the batch between backward calls */
struct AdjScratch {
  size_t cap_vertices = 0;
  void *mem = nullptr;
  AdjQ *d_qs = nullptr;
  AdjG *d_gs = nullptr;
  unsigned *d_qidx = nullptr;
  unsigned *d_flag = nullptr;
  void *d_hand = nullptr;
  size_t cap_hand = 0;
  size_t nq = 0, ng = 0;
};

void adds_adjoint_free(void *p) {
  AdjScratch *s = (AdjScratch *)p;
  if (!s) return;
  if (s->mem) cudaFree(s->mem);
  if (s->d_qs) cudaFree(s->d_qs);
  if (s->d_gs) cudaFree(s->d_gs);
  if (s->d_qidx) cudaFree(s->d_qidx);
  if (s->d_flag) cudaFree(s->d_flag);
  if (s->d_hand) cudaFree(s->d_hand);
  delete s;
}

static int adj_fail(cudaError_t e) {
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? ADDS_ERR_OOM : ADDS_ERR_CUDA;
}
#define CKA(x)                                  \
  do {                                          \
    cudaError_t _e = (x);                       \
    if (_e != cudaSuccess) return adj_fail(_e); \
  } while (0)

/* Core: queries (row, edges, n, src, dist, seed) + graphs (edges, m, grad,
 * query list) -> gradient. */
static int run_adjoint(AdjScratch *S, std::vector<AdjQ> &qh, std::vector<AdjG> &gh,
                       const std::vector<unsigned> &qidx, unsigned max_deg, int accumulate,
                       cudaStream_t st) {
  size_t need = 0;
  unsigned max_n = 0;
  for (auto &q : qh) {
    need += ((size_t)q.n + 31) & ~(size_t)31;
    if (q.n > max_n) max_n = q.n;
  }
  if (need > S->cap_vertices) {
    if (S->mem) cudaFree(S->mem);
    S->mem = nullptr;
    CKA(cudaMalloc(&S->mem, need * 24));
    S->cap_vertices = need;
  }
  if (qh.size() != S->nq) {
    if (S->d_qs) cudaFree(S->d_qs);
    S->d_qs = nullptr;
    CKA(cudaMalloc(&S->d_qs, qh.size() * sizeof(AdjQ)));
    S->nq = qh.size();
  }
  if (gh.size() != S->ng) {
    if (S->d_gs) cudaFree(S->d_gs);
    if (S->d_qidx) cudaFree(S->d_qidx);
    S->d_gs = nullptr;
    S->d_qidx = nullptr;
    CKA(cudaMalloc(&S->d_gs, gh.size() * sizeof(AdjG)));
    CKA(cudaMalloc(&S->d_qidx, qidx.size() * sizeof(unsigned)));
    S->ng = gh.size();
  }
  if (!S->d_flag) CKA(cudaMalloc(&S->d_flag, 16));
  /* carve: pred u64 | lam u64 | kids | round */
  unsigned long long *pred = (unsigned long long *)S->mem;
  unsigned long long *lam = pred + need;
  unsigned *kids = (unsigned *)(lam + need);
  unsigned *round = kids + need;
  size_t off = 0;
  unsigned long long tiles = 0, etiles = 0;
  for (auto &q : qh) {
    q.pred = pred + off;
    q.lam = lam + off;
    q.kids = kids + off;
    q.round = round + off;
    off += ((size_t)q.n + 31) & ~(size_t)31;
    q.tile0 = (unsigned)tiles;
    tiles += (q.n + adj::TILE - 1u) / adj::TILE;
  }
  for (auto &g : gh) {
    g.tile0 = (unsigned)etiles;
    etiles += ((unsigned long long)g.m + adj::TILE - 1u) / adj::TILE;
  }
  /* HAND walks of each of a tile's 4 warps */
  const size_t hands = (size_t)tiles * 4u * adj::HAND;
  if (hands > S->cap_hand) {
    if (S->d_hand) cudaFree(S->d_hand);
    S->d_hand = nullptr;
    S->cap_hand = 0;
    CKA(cudaMalloc(&S->d_hand, hands * sizeof(adj::Walk)));
    S->cap_hand = hands;
  }
  if (tiles > 0x7FFFFFFFull || etiles > 0x7FFFFFFFull) return ADDS_ERR_UNSUPPORTED;
  CKA(cudaMemcpyAsync(S->d_qs, qh.data(), qh.size() * sizeof(AdjQ), cudaMemcpyHostToDevice, st));
  CKA(cudaMemcpyAsync(S->d_gs, gh.data(), gh.size() * sizeof(AdjG), cudaMemcpyHostToDevice, st));
  CKA(cudaMemcpyAsync(S->d_qidx, qidx.data(), qidx.size() * sizeof(unsigned),
                      cudaMemcpyHostToDevice, st));
  const unsigned nq = (unsigned)qh.size(), ng = (unsigned)gh.size(), T = (unsigned)tiles;
  auto children = [&] {
    if (max_deg <= 32u) adj::k_children<true><<<T, 256, 0, st>>>(S->d_qs, nq, S->d_flag);
    else adj::k_children<false><<<T, 256, 0, st>>>(S->d_qs, nq, S->d_flag);
  };
  adj::k_init<<<T, 256, 0, st>>>(S->d_qs, nq);
  adj::k_pred_strict<<<T, 256, 0, st>>>(S->d_qs, nq);
  CKA(cudaMemsetAsync(S->d_flag, 0, 8, st));
  children();
  unsigned orphans = 0;
  CKA(cudaMemcpyAsync(&orphans, S->d_flag, 4, cudaMemcpyDeviceToHost, st));
  CKA(cudaStreamSynchronize(st));
  if (orphans) { /* zero-gap ties */
    adj::k_rounds_init<<<T, 256, 0, st>>>(S->d_qs, nq);
    for (unsigned r = 1; r <= max_n; ++r) {
      unsigned changed = 0;
      CKA(cudaMemsetAsync(S->d_flag, 0, 4, st));
      adj::k_pred_zero<<<T, 256, 0, st>>>(S->d_qs, nq, r, S->d_flag);
      CKA(cudaMemcpyAsync(&changed, S->d_flag, 4, cudaMemcpyDeviceToHost, st));
      CKA(cudaStreamSynchronize(st));
      if (!changed) break;
    }
    children();
  }
  if (T >= 8u * 148u) {
    adj::Walk *hand = (adj::Walk *)S->d_hand;
    unsigned *ctr = S->d_flag + 2;
    CKA(cudaMemsetAsync(ctr, 0, 8, st));
    if (max_deg <= 32u) {
      adj::k_walk<true, true, true><<<T, 128, 0, st>>>(S->d_qs, nq, hand, ctr);
      adj::k_walk<true, false, false><<<148 * 12, 128, 0, st>>>(S->d_qs, nq, hand, ctr);
    } else {
      adj::k_walk<false, true, true><<<T, 128, 0, st>>>(S->d_qs, nq, hand, ctr);
      adj::k_walk<false, false, false><<<148 * 12, 128, 0, st>>>(S->d_qs, nq, hand, ctr);
    }
  } else { /* too few tiles to fill the SMs: nothing to make room for */
    if (max_deg <= 32u) adj::k_walk<true, true, false><<<T, 512, 0, st>>>(S->d_qs, nq, nullptr, nullptr);
    else adj::k_walk<false, true, false><<<T, 512, 0, st>>>(S->d_qs, nq, nullptr, nullptr);
  }
  if (etiles)
    adj::k_grad<<<(unsigned)etiles, 256, 0, st>>>(S->d_gs, ng, S->d_qs, S->d_qidx, accumulate);
  CKA(cudaGetLastError());
  CKA(cudaStreamSynchronize(st));
  return ADDS_OK;
}

extern "C" int adds_batch_backward(adds_batch *b, const float *const *grad_dist,
                                   float *const *grad_w) {
  if (!b || !grad_dist || !grad_w) return ADDS_ERR_INVALID;
  cudaStream_t st;
  unsigned nq;
  std::vector<adds_graph *> *qgraph, *ugraph;
  std::vector<uint32_t> *srcs;
  std::vector<unsigned> *qgid;
  unsigned *dist_all;
  std::vector<size_t> *dist_off;
  void **adjp;
  adds_batch_internal(b, &st, &nq, &qgraph, &srcs, &ugraph, &qgid, &dist_all, &dist_off, &adjp);
  const unsigned *row;
  const uint2 *edges;
  uint32_t n;
  uint64_t m;
  unsigned deg, max_deg = 0;
  int dev;
  adds_graph_internal((*qgraph)[0], &row, &edges, &n, &m, &deg, &dev);
  CKA(cudaSetDevice(dev));
  std::vector<AdjQ> qh(nq);
  for (unsigned i = 0; i < nq; ++i) {
    adds_graph_internal((*qgraph)[i], &row, &edges, &n, &m, &deg, &dev);
    AdjQ q;
    memset(&q, 0, sizeof q);
    q.row = row;
    q.edges = edges;
    q.dist = (const float *)(dist_all + (*dist_off)[i]);
    q.seed = grad_dist[i];
    q.n = n;
    q.src = (*srcs)[i];
    qh[i] = q;
  }
  std::vector<AdjG> gh(ugraph->size());
  std::vector<unsigned> qidx;
  for (size_t gi = 0; gi < ugraph->size(); ++gi) {
    adds_graph_internal((*ugraph)[gi], &row, &edges, &n, &m, &deg, &dev);
    if (!grad_w[gi]) return ADDS_ERR_INVALID;
    AdjG g;
    max_deg = std::max(max_deg, deg);
    g.edges = edges;
    g.m = (unsigned)m;
    g.grad = grad_w[gi];
    g.q_begin = (unsigned)qidx.size();
    for (unsigned i = 0; i < nq; ++i)
      if ((*qgid)[i] == gi) qidx.push_back(i);
    g.q_end = (unsigned)qidx.size();
    gh[gi] = g;
  }
  if (!*adjp) *adjp = new AdjScratch();
  return run_adjoint((AdjScratch *)*adjp, qh, gh, qidx, max_deg, 1, st);
}

extern "C" int adds_sssp_backward(adds_graph *g, uint32_t ns, const uint32_t *srcs, const float *dist,
                                  const float *grad_dist, float *grad_w, const adds_opts *opts) {
  if (!g || !srcs || !dist || !grad_w || ns == 0) return ADDS_ERR_INVALID;
  const unsigned *row;
  const uint2 *edges;
  uint32_t n;
  uint64_t m;
  unsigned deg;
  int dev;
  adds_graph_internal(g, &row, &edges, &n, &m, &deg, &dev);
  for (uint32_t i = 0; i < ns; ++i)
    if (srcs[i] >= n) return ADDS_ERR_INVALID;
  CKA(cudaSetDevice(dev));
  cudaStream_t st = (opts && opts->stream) ? (cudaStream_t)opts->stream : 0;
  std::vector<AdjQ> qh(ns);
  std::vector<unsigned> qidx(ns);
  for (uint32_t i = 0; i < ns; ++i) {
    AdjQ q;
    memset(&q, 0, sizeof q);
    q.row = row;
    q.edges = edges;
    q.dist = dist + (size_t)i * n;
    q.seed = grad_dist ? grad_dist + (size_t)i * n : nullptr;
    q.n = n;
    q.src = srcs[i];
    qh[i] = q;
    qidx[i] = i;
  }
  std::vector<AdjG> gh(1);
  gh[0].edges = edges;
  gh[0].m = (unsigned)m;
  gh[0].grad = grad_w;
  gh[0].q_begin = 0;
  gh[0].q_end = ns;
  AdjScratch S;
  const int rc = run_adjoint(&S, qh, gh, qidx, deg, 0, st);
  if (S.mem) cudaFree(S.mem);
  if (S.d_qs) cudaFree(S.d_qs);
  if (S.d_gs) cudaFree(S.d_gs);
  if (S.d_qidx) cudaFree(S.d_qidx);
  if (S.d_flag) cudaFree(S.d_flag);
  if (S.d_hand) cudaFree(S.d_hand);
  return rc;
}
