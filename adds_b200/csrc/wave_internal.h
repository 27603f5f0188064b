/*
 * wave_internal.h — device data layout of the wave kernels (wave.cu).
 *
 * One group (a CTA, or several that exchange) solves one query with two
 * kinds of lists: the frontier of the current step, kept in shared memory
 * with an overflow area in HBM, and a far list per CTA in HBM.  No page
 * pool, no bucket ring, no barrier through memory.
 */
#ifndef ADDS_WAVE_INTERNAL_H_
#define ADDS_WAVE_INTERNAL_H_

#include <cuda_runtime.h>
#include <stdint.h>

/* error word of a launch (first one wins) */
#define WV_ERR_OVERFLOW 1u /* a list outgrew its area: solve on another engine */
#define WV_ERR_TIMEOUT 2u
#define WV_ERR_INPUT 3u    /* nothing to solve: the caller's arrays are invalid   */

#define WV_SETTLED 4u     /* in a note: the CTA holds settled entries           */
#define WV_NOTE_BITS 3u   /* a note's error code and WV_SETTLED                 */
#define WV_PIECE 512u     /* edges of a long row one entry stands for          */
#define WV_MAX_GROUP 160u /* CTAs of one group (a multiple of 32)              */
/* a group's two sets of 16-byte notes, and (after all groups' notes) two sets
 * of 32 bytes on the settled entries */
#define WV_GRP_WORDS (2u * (4u + 8u) * WV_MAX_GROUP)

/* Two notes' states as one: the larger error code, since codes are numbers
 * (overflow and timeout side by side are a timeout, not their OR, bad input),
 * and whether any CTA holds settled entries. */
static __host__ __device__ inline unsigned wv_worse(unsigned a, unsigned b) {
  const unsigned ea = a & (WV_SETTLED - 1u), eb = b & (WV_SETTLED - 1u);
  return (ea > eb ? ea : eb) | ((a | b) & WV_SETTLED);
}

struct WvQuery {
  const unsigned *row;
  const uint2 *edges; /* rows in CSR order, or sorted by weight where split is  */
  const unsigned *split; /* WV_POOL: light edges (w < delta) at the start of each
                            row; null: every row is relaxed whole             */
  /* in-edges (the transposed graph, {tail, weight}) and the smallest heavy
   * weight's bits, where heavy edges may be pulled; else null                */
  const unsigned *trow;
  const uint2 *tedges;
  /* rows of more than WV_PIECE edges: their first piece by vertex, and the
   * pieces {vertex, first edge, edges, 0}; null where no row is that long */
  const unsigned *first;
  const uint4 *piece;
  unsigned *dist;
  unsigned n;
  unsigned src;
  float delta;        /* first step of the near threshold, in distance units   */
  unsigned np;        /* pieces                                               */
  unsigned thr;
  unsigned hops;      /* groups: hops between two exchanges                   */
  unsigned grow;      /* groups: the threshold's step may widen               */
  unsigned long long m;
};

/* list areas of one CTA, in 8-byte entries from WvParams::ws */
struct WvArea {
  unsigned long long off; /* two frontier overflow areas, then the far list    */
  unsigned ncap, fcap;    /* entries of one frontier overflow area / far list  */
  unsigned scap, pad;     /* entries of the settled list                       */
};

struct WvStat {
  unsigned err;           /* kept until the host resets the engine             */
  unsigned pad0[31];
  unsigned next;          /* batch: next query (in order) to take              */
  unsigned pad1[31];
  unsigned long long items, stale, edges, pushes, steps, splits;
};

struct WvParams {
  const WvQuery *qs;
  const unsigned *order;  /* the queries, largest first                        */
  const unsigned *qoff;   /* [groups + 1]: each group's share of the order; null:
                             one group, or (one CTA per query) all of it       */
  unsigned nq, groups, gsize; /* queries, groups of CTAs, CTAs of one        */
  const WvArea *area;     /* [groups * gsize]                                  */
  void *ws;
  WvStat *st;
  unsigned *grp;          /* a group's notes, two sets; cleared before a launch */
  unsigned single_src;    /* overrides query 0's source when != ~0             */
  unsigned filled;        /* the distances hold INF and the source already     */
  unsigned low;           /* a frontier below this takes more far entries      */
  unsigned high;          /* a frontier above this narrows the threshold step  */
  unsigned long long timeout_ns;
};

#ifdef __cplusplus
#include <vector>

struct WvEngine {
  int device = -1;
  bool flt = false;
  int shape = -1;         /* variant asked for                                  */
  int kernel = -1;        /* variant launched (WV_PULL for WV_POOL with in-edges) */
  unsigned nq = 0, groups = 0, gsize = 1, ctas = 0, req_gsize = 0;
  unsigned *grp = nullptr;
  WvQuery *qs = nullptr;
  unsigned *order = nullptr;
  WvArea *area = nullptr;
  void *ws = nullptr;
  WvStat *st = nullptr;
  WvStat *st_host = nullptr; /* pinned                                         */
  std::vector<WvQuery> qs_host;
  bool shares = false;  /* order is split over the groups                       */
  bool fills = false;   /* the last launch was preceded by the fill kernel     */
  bool has_set = false; /* room for settled lists                             */
  size_t bytes = 0;
};

/* kernel variants: one CTA per query (256 or 1,024 threads), a group of CTAs,
 * a group whose CTAs pool the edges of their entries */
#define WV_CTA 0
#define WV_WIDE 1
#define WV_GROUP 2
#define WV_POOL 3
#define WV_PULL 4 /* WV_POOL with queries that have in-edges                    */
#define WV_LAST WV_POOL

/* the kernels themselves (noalloc.cu brings its own memory): residency of a
 * variant (needed before its first launch), the schedule's parameters for P's
 * group size, a launch, and a CTA's frontier entries in shared memory */
cudaError_t wv_prepare(bool flt, int shape, int *ctas_per_sm);
void wv_schedule(WvParams &P, int shape);
void wv_query_schedule(WvQuery &q, int shape);
cudaError_t wv_launch(const WvParams &P, bool flt, int shape, cudaStream_t st);
unsigned wv_near(int shape);

int wv_engine_alloc(WvEngine &E, int device, bool flt, int shape, unsigned gsize,
                    const std::vector<WvQuery> &qv, cudaStream_t st);
void wv_engine_free(WvEngine &E);
int wv_engine_reset(WvEngine &E, cudaStream_t st);
int wv_engine_upload(WvEngine &E, cudaStream_t st);
int wv_engine_enqueue(WvEngine &E, unsigned single_src, unsigned long long timeout_ns,
                      cudaStream_t st, cudaEvent_t k0, cudaEvent_t k1);
int wv_engine_status(const WvEngine &E, char *msg, size_t msg_len);
#endif

#endif /* ADDS_WAVE_INTERNAL_H_ */
