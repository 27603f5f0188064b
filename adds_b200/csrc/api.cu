/*
 * api.cu — host side of the C ABI (include/adds.h).
 *
 * Replaces the reference host driver gg_main (ads_int/kernel.cu:185-288) and
 * the host half of the worklist (wl.h:203-460): sizing and allocation of the
 * bucket pool, per-solve reset, the delta choice (profiler_kernel + set_param,
 * kernel.cu:153-183 / wl.h:395-449), the launch, timing, and the work count.
 * Differences by design: errors are return codes (no exit/assert), the pool
 * regrows and the solve reruns when the device reports overflow, and the
 * launch is one cooperative persistent kernel instead of CDP children.
 */
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <errno.h>
#include <fcntl.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <thread>
#include <vector>

#include "../../include/adds.h"
#include "adds_internal.h"
#include "phase_internal.h"
#include "wave_internal.h"

/* engine.cu */
cudaError_t adds_engine_prepare(bool flt, int block, int *max_blocks_per_sm);
cudaError_t adds_engine_launch_init(const EngParams &P, unsigned max_n, cudaStream_t st);
cudaError_t adds_engine_launch_solve(const EngParams &P, int block, cudaStream_t st);
cudaError_t adds_engine_launch_reached(const unsigned *row, const unsigned *dist, unsigned n,
                                       unsigned inf, unsigned long long *out, cudaStream_t st);
cudaError_t adds_engine_launch_reset(unsigned long long *fq, unsigned fq_cells,
                                     unsigned pool_pages, unsigned *hub_seq, unsigned hub_cells,
                                     cudaStream_t st);
/* gen.cu */
int adds_gen_build(const adds_gen_spec *sp, unsigned **row_out, uint2 **edges_out,
                   uint32_t *n_out, uint64_t *m_out, cudaStream_t st);
/* adjoint.cu */
int adds_adjoint_run(struct AdjointJob *job);

/* ------------------------------------------------------------------------ */
static thread_local char g_last_err[256] = "";

static int cuda_fail(cudaError_t e, const char *what) {
  snprintf(g_last_err, sizeof g_last_err, "%s: %s", what, cudaGetErrorString(e));
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return ADDS_ERR_OOM;
  }
  cudaGetLastError();
  return ADDS_ERR_CUDA;
}
#define CK(x)                                      \
  do {                                             \
    cudaError_t _e = (x);                          \
    if (_e != cudaSuccess) return cuda_fail(_e, #x); \
  } while (0)

/* diagnostics text for adds_last_cuda_error (used by noalloc.cu too) */
void adds_set_last_error(const char *msg) { snprintf(g_last_err, sizeof g_last_err, "%s", msg); }

extern "C" int adds_abi_version(void) { return ADDS_ABI_VERSION; }
extern "C" const char *adds_last_cuda_error(void) { return g_last_err; }

extern "C" const char *adds_strerror(int code) {
  switch (code) {
    case ADDS_OK: return "ok";
    case ADDS_ERR_INVALID: return "invalid argument";
    case ADDS_ERR_IO: return "i/o error";
    case ADDS_ERR_FORMAT: return "malformed graph file";
    case ADDS_ERR_OOM: return "out of memory";
    case ADDS_ERR_CUDA: return "CUDA runtime error";
    case ADDS_ERR_DEVICE_TIMEOUT: return "bounded device wait timed out";
    case ADDS_ERR_WL_OVERFLOW: return "worklist pool exhausted";
    case ADDS_ERR_NO_DEVICE: return "no usable sm_100 device";
    case ADDS_ERR_UNSUPPORTED: return "unsupported request";
    default: return "unknown error";
  }
}

extern "C" void adds_opts_init(adds_opts *o) {
  if (!o) return;
  memset(o, 0, sizeof *o);
  o->delta_shift = -1;
  o->delta_scale = 0.f;
  o->adapt = -1;
  o->strict_order = -1;
  o->local_max = -1;
  o->light_heavy = -1;
  o->block_threads = 0;
  o->greed = -1;
  o->engine = ADDS_ENGINE_AUTO;
  o->group_ctas = 0;
  o->solo_max = -1;
}

static unsigned next_pow2(unsigned long long x) {
  unsigned l = 0;
  while ((1ull << l) < x) ++l;
  return l;
}

/* ------------------------------------------------------------------------ */
/* engine: the bucket pool and per-query queue state                         */
struct EngQuery {
  const unsigned *row;
  const uint2 *edges;
  const unsigned *split;
  unsigned *dist;
  unsigned n;
  unsigned long long m;
  unsigned src;
  float scale;
  unsigned shift;
  unsigned graph_id;
};

struct Engine {
  int device = -1;
  bool flt = false;
  unsigned nq = 0;
  unsigned pool_pages = 0, fq_cells = 0, max_n = 0;
  unsigned long long *pool = nullptr;
  unsigned *pgen = nullptr, *pcons = nullptr;
  unsigned long long *fq = nullptr;
  HubChunk *hub = nullptr;
  unsigned *hub_seq = nullptr;
  GlobalCtl *g = nullptr;
  QueryDesc *qs = nullptr;
  QueryCtl *ctl = nullptr;
  SlotCtr *slots = nullptr;
  unsigned long long *pt = nullptr;
  unsigned long long *reach = nullptr;
  GlobalCtl *g_host = nullptr; /* pinned */
  std::vector<QueryDesc> qs_host;
  size_t bytes = 0;
  int max_bps[3] = {0, 0, 0}; /* resident CTAs per SM for 128/256/512 threads */
  int num_sms = 0;
};

static int block_index(int block) { return block == 128 ? 0 : (block == 256 ? 1 : 2); }

static void engine_free(Engine &E) {
  void *ptrs[] = {E.pool, E.pgen, E.pcons, E.fq, E.hub, E.hub_seq, E.g, E.qs, E.ctl, E.slots, E.pt, E.reach};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (E.g_host) cudaFreeHost(E.g_host);
  E = Engine();
}

static int engine_full_reset(Engine &E, cudaStream_t st) {
  const unsigned hub_cells = 1u << ADDS_HUB_RING_LOG2;
  CK(cudaMemsetAsync(E.pool, 0, (size_t)E.pool_pages * ADDS_PAGE * 8, st));
  CK(cudaMemsetAsync(E.pgen, 0, (size_t)E.pool_pages * 4, st));
  CK(cudaMemsetAsync(E.pcons, 0, (size_t)E.pool_pages * 4, st));
  CK(cudaMemsetAsync(E.g, 0, sizeof(GlobalCtl), st));
  CK(cudaMemsetAsync(E.slots, 0, (size_t)E.nq * 2 * ADDS_NB * sizeof(SlotCtr), st));
  CK(cudaMemsetAsync(E.ctl, 0, (size_t)E.nq * sizeof(QueryCtl), st));
  size_t pt_words = 0;
  for (auto &q : E.qs_host) pt_words += (size_t)2 * ADDS_NB << q.ptn_log2;
  CK(cudaMemsetAsync(E.pt, 0xFF, pt_words * 8, st));
  const unsigned long long tail = E.pool_pages;
  CK(cudaMemcpyAsync(&E.g->fq_tail, &tail, 8, cudaMemcpyHostToDevice, st));
  CK(adds_engine_launch_reset(E.fq, E.fq_cells, E.pool_pages, E.hub_seq, hub_cells, st));
  CK(cudaStreamSynchronize(st));
  return ADDS_OK;
}

static int engine_upload_queries(Engine &E, cudaStream_t st) {
  CK(cudaMemcpyAsync(E.qs, E.qs_host.data(), E.qs_host.size() * sizeof(QueryDesc),
                     cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));
  return ADDS_OK;
}

/* Sizes the pool for the queries (x grow) and allocates everything. */
static int engine_alloc(Engine &E, int device, bool flt, const std::vector<EngQuery> &qv,
                        unsigned grow, cudaStream_t st) {
  engine_free(E);
  E.device = device;
  E.flt = flt;
  E.nq = (unsigned)qv.size();
  for (int i = 0; i < 3; ++i) {
    CK(adds_engine_prepare(flt, 128 << i, &E.max_bps[i]));
    if (E.max_bps[i] < 1) return ADDS_ERR_UNSUPPORTED; /* variant cannot be resident */
  }
  CK(cudaDeviceGetAttribute(&E.num_sms, cudaDevAttrMultiProcessorCount, device));
  if (E.num_sms < 1) return ADDS_ERR_UNSUPPORTED;
  double sum_need = 0;
  E.qs_host.resize(E.nq);
  size_t pt_words = 0;
  for (unsigned i = 0; i < E.nq; ++i) {
    const EngQuery &q = qv[i];
    const double need = 3.0 * q.n + q.m / 8.0 + 64.0;
    sum_need += need;
    unsigned ptl = next_pow2((unsigned long long)(need * grow / ADDS_PAGE) + 8ull);
    if (ptl < 4) ptl = 4;
    QueryDesc d;
    memset(&d, 0, sizeof d);
    d.row = q.row;
    d.edges = q.edges;
    d.split = q.split;
    d.dist = q.dist;
    d.n = q.n;
    d.src = q.src;
    d.scale = q.scale;
    d.ptn_log2 = ptl;
    d.shift0 = q.shift;
    d.graph_id = q.graph_id;
    E.qs_host[i] = d;
    pt_words += (size_t)2 * ADDS_NB << ptl;
    if (q.n > E.max_n) E.max_n = q.n;
  }
  unsigned long long pages = (unsigned long long)(sum_need * grow / ADDS_PAGE) + 2ull * ADDS_NB * E.nq + 64ull;
  if (pages > 0x7FFFFFF0ull) return ADDS_ERR_OOM;
  E.pool_pages = (unsigned)pages;
  E.fq_cells = 1u << next_pow2(pages);
  const unsigned hub_cells = 1u << ADDS_HUB_RING_LOG2;
#define ALLOC(ptr, bytes_)                                          \
  do {                                                              \
    size_t _b = (bytes_);                                           \
    cudaError_t _e = cudaMalloc((void **)&(ptr), _b);               \
    if (_e != cudaSuccess) {                                        \
      int _rc = cuda_fail(_e, "engine alloc " #ptr);                \
      engine_free(E);                                               \
      return _rc;                                                   \
    }                                                               \
    E.bytes += _b;                                                  \
  } while (0)
  ALLOC(E.pool, (size_t)E.pool_pages * ADDS_PAGE * 8);
  ALLOC(E.pgen, (size_t)E.pool_pages * 4);
  ALLOC(E.pcons, (size_t)E.pool_pages * 4);
  ALLOC(E.fq, (size_t)E.fq_cells * 8);
  ALLOC(E.hub, (size_t)hub_cells * sizeof(HubChunk));
  ALLOC(E.hub_seq, (size_t)hub_cells * 4);
  ALLOC(E.g, sizeof(GlobalCtl));
  ALLOC(E.qs, (size_t)E.nq * sizeof(QueryDesc));
  ALLOC(E.ctl, (size_t)E.nq * sizeof(QueryCtl));
  ALLOC(E.slots, (size_t)E.nq * 2 * ADDS_NB * sizeof(SlotCtr));
  ALLOC(E.pt, pt_words * 8);
  ALLOC(E.reach, 16);
#undef ALLOC
  if (cudaMallocHost((void **)&E.g_host, sizeof(GlobalCtl)) != cudaSuccess) {
    cudaGetLastError();
    engine_free(E);
    return ADDS_ERR_OOM;
  }
  size_t off = 0;
  for (unsigned i = 0; i < E.nq; ++i) {
    E.qs_host[i].pt = E.pt + off;
    off += (size_t)2 * ADDS_NB << E.qs_host[i].ptn_log2;
    E.qs_host[i].slots = E.slots + (size_t)i * 2 * ADDS_NB;
    E.qs_host[i].ctl = E.ctl + i;
  }
  int rc = engine_upload_queries(E, st);
  if (rc) return rc;
  return engine_full_reset(E, st);
}

/* resolved knobs */
struct Knobs {
  int window, ctas_per_sm, batch_max, hub_threshold, hub_chunk, strict, adapt, local_max,
      light_heavy, block, greed;
  int engine, variant, group_ctas, solo_max, near_far, dense_scan; /* phase engine */
  int pull; /* phase engine: heavy phases may run as a pull (in-edge CSR)     */
  int wave; /* wave kernel variant (WV_*) that solves instead of an engine, or -1 */
  unsigned long long timeout_ns;
};

/* phase-engine kernel variant for threads per CTA (the CTAs per SM follow
 * from its shared memory) */
static int phase_variant(int block, int cps) {
  if (block == 1024) return 2;
  if (block == 512) return cps == 1 ? 4 : 1;
  if (block == 128) return 5;
  return cps == 2 ? 3 : 0;
}

static PhKnobs phase_knobs(const Knobs &k) {
  PhKnobs p;
  p.variant = k.variant;
  p.ctas_per_sm = 0;
  p.group_ctas = k.group_ctas;
  p.hub_threshold = (unsigned)std::max(64, k.hub_threshold);
  p.hub_chunk = 1024u;
  p.solo_max = (unsigned)std::max(0, k.solo_max);
  p.adapt = k.adapt > 0 ? 1u : 0u;
  p.lh_adapt = k.light_heavy == 2 ? 1u : 0u;
  p.near_far = k.near_far ? 1u : 0u;
  p.dense_shift = (k.dense_scan > 0 && !k.near_far) ? (unsigned)std::min(k.dense_scan, 31) : 0u;
  p.timeout_ns = k.timeout_ns;
  return p;
}

static EngParams make_params(const Engine &E, const Knobs &k, unsigned single_src) {
  EngParams P;
  memset(&P, 0, sizeof P);
  P.qs = E.qs;
  P.nq = E.nq;
  const int blk = (k.block == 128 || k.block == 256 || k.block == 512) ? k.block : 256;
  const int maxb = E.max_bps[block_index(blk)];
  int cps = k.ctas_per_sm;
  if (cps <= 0 || cps > maxb) cps = maxb;
  P.nctas = (unsigned)(cps * E.num_sms);
  P.block = (unsigned)blk;
  P.greed = (unsigned)std::max(0, std::min(k.greed, 12));
  P.g = E.g;
  P.pool = E.pool;
  P.pgen = E.pgen;
  P.pcons = E.pcons;
  P.fq = E.fq;
  P.fq_mask = E.fq_cells - 1u;
  P.pool_pages = E.pool_pages;
  P.hub = E.hub;
  P.hub_seq = E.hub_seq;
  P.timeout_ns = k.timeout_ns;
  P.alloc_wait_ns = 200ull * 1000ull * 1000ull;
  if (P.alloc_wait_ns > k.timeout_ns) P.alloc_wait_ns = k.timeout_ns;
  P.window = (unsigned)std::max(1, std::min(k.window, ADDS_NB));
  P.batch_max = (unsigned)std::max(1, std::min(k.batch_max, blk));
  P.hub_threshold = (unsigned)std::max(k.hub_threshold, 64);
  P.hub_chunk = (unsigned)std::max(k.hub_chunk, 64);
  if (P.hub_chunk > P.hub_threshold) P.hub_chunk = P.hub_threshold;
  P.strict_order = (unsigned)k.strict;
  P.adapt = (unsigned)k.adapt;
  P.is_float = E.flt ? 1u : 0u;
  P.single_src = single_src;
  P.local_max = (unsigned)std::max(0, std::min(k.local_max, blk));
  P.local_max_hungry = P.local_max / 8u;
  return P;
}

static int engine_enqueue(Engine &E, const EngParams &P, cudaStream_t st,
                          cudaEvent_t k0 = nullptr, cudaEvent_t k1 = nullptr) {
  /* under stream capture the records must be external nodes to stay
   * usable for timing; outside capture the flag is not allowed */
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(st, &cs));
  const unsigned fl = cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : 0u;
  CK(adds_engine_launch_init(P, E.max_n, st));
  if (k0) CK(cudaEventRecordWithFlags(k0, st, fl));
  CK(adds_engine_launch_solve(P, (int)P.block, st));
  if (k1) CK(cudaEventRecordWithFlags(k1, st, fl));
  CK(cudaMemcpyAsync(E.g_host, E.g, sizeof(GlobalCtl), cudaMemcpyDeviceToHost, st));
  return ADDS_OK;
}

/* device error word -> ABI code (after the stream has been synchronised) */
static int engine_status(const Engine &E) {
  if (E.g_host->err)
    snprintf(g_last_err, sizeof g_last_err, "device error %u at wait site %u", E.g_host->err,
             E.g_host->err_where);
  switch (E.g_host->err) {
    case ADDS_DEV_OK: return ADDS_OK;
    case ADDS_DEV_OVERFLOW: return ADDS_ERR_WL_OVERFLOW;
    case ADDS_DEV_HUB_OVERFLOW: return ADDS_ERR_WL_OVERFLOW;
    default: return ADDS_ERR_DEVICE_TIMEOUT;
  }
}

static void fill_stats(const Engine &E, const EngParams &P, adds_stats *s) {
  if (!s) return;
  const GlobalCtl &g = *E.g_host;
  s->items_popped = g.st_items;
  s->items_stale = g.st_stale;
  s->edges_scanned = g.st_edges;
  s->pushes = g.st_pushes;
  s->batches = g.st_batches;
  s->hub_chunks = g.st_hub;
  s->hub_stale = g.st_hub_stale;
  s->local_batches = g.st_local;
  s->heavy_lists = g.st_heavy;
  for (int i = 0; i < 6; ++i) s->phase_cycles[i] = g.st_cyc[i];
  s->mid_flush_cycles = g.st_pad[0];
  s->mid_flushes = g.st_pad[1];
  s->ctas = (int32_t)P.nctas;
  s->launches = 2; /* init kernel, persistent solver */
}

/* ------------------------------------------------------------------------ */
/* graphs                                                                     */

/* Where the light edges of each sorted row end, for one bucket width.  A graph's
 * plain solves and each of its batches own one: their widths differ, they may
 * run at the same time, and a pull relies on its solve's own threshold. */
struct Split {
  unsigned *at = nullptr; /* light-edge count per row                       */
  unsigned thr = 0;       /* ... of weights below this (weight bits)        */
  unsigned long long wversion = 0; /* ... of these weights                  */
  bool valid = false;
};

struct adds_graph {
  int device = 0;
  adds_wtype wt = ADDS_I32;
  uint32_t n = 0;
  uint64_t m = 0;
  unsigned *row = nullptr;
  uint2 *edges = nullptr;
  unsigned *dist = nullptr;
  uint2 *sedges = nullptr;     /* rows sorted by weight (light edges first)   */
  bool sorted_valid = false;
  Split split;                 /* the plain solves' one                       */
  unsigned *trow = nullptr;    /* in-edge CSR (pull phases): n+1 offsets      */
  uint2 *tedges = nullptr;     /* {tail vertex, weight bits} per in-edge      */
  bool trans_valid = false;
  unsigned long long wversion = 0; /* bumped by adds_graph_set_weights */
  void *sw_jobs = nullptr;        /* adds_graphs_set_weights' descriptors      */
  size_t sw_cap = 0;
  unsigned *aux = nullptr;        /* 64 B: validation flag + weight sample sum */
  uint32_t *sort_buf = nullptr;   /* 4*m words: keys/values in and out          */
  void *sort_tmp = nullptr;
  size_t sort_tmp_bytes = 0;
  cudaStream_t stream = nullptr;
  uint32_t max_deg = 0;
  double avg_deg = 0, avg_w = 0;
  size_t bytes = 0;
  Engine eng;
  PhEngine peng;       /* phase engine (allocated on first use)            */
  WvEngine weng;       /* wave kernels (allocated on first use)            */
  /* Their lists overflowed on this graph, or found no memory.  For good: how
   * much is pending at once follows from its shape more than from the source
   * or the weights, and each new try would cost the lists and a lost solve. */
  bool wave_off = false;
  unsigned *wfirst = nullptr; /* pieces of long rows (WvQuery)              */
  uint4 *wpiece = nullptr;
  unsigned wpieces = 0;
  unsigned trace_cap = 0; /* phase trace records requested (0 = off)       */
  PhParams last_pp;
  int last_engine = 0; /* engine of the solves in flight                   */
  bool last_wave = false; /* ... which the wave kernels run                */
  int last_shift = 0;     /* ... with this bucket shift                    */
  unsigned grow = 1;
  int tuned = 0;
  adds_opts tuned_opts; /* the fastest engine's knobs                         */
  adds_opts tuned_wave; /* the wave kernel that beat it, as it was timed (wave
                           0: none did)                                      */
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  Knobs last_knobs;
  EngParams last_params;
  int pending = 0; /* async solves enqueued since the last sync */
  /* their sources and options: adds_graph_sync runs them again, on a grown
   * worklist pool, when one of them ran out of worklist space */
  std::vector<std::pair<uint32_t, adds_opts>> pend;
  /* adds_sssp_sources: two staging copies of dist, the copy-out stream and
   * its events (made on first use) */
  unsigned *stage = nullptr;
  cudaStream_t cstream = nullptr;
  cudaEvent_t ev_ready[2] = {nullptr, nullptr}, ev_free[2] = {nullptr, nullptr};
  /* per-solve event ring: (start, kernel start, kernel end, end) */
  static constexpr int kRing = 256;
  cudaEvent_t ring[kRing][4] = {};
  int ring_used = 0;
};

static int set_device(int dev) {
  int cnt = 0;
  if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
    cudaGetLastError();
    return ADDS_ERR_NO_DEVICE;
  }
  if (dev < 0 || dev >= cnt) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(dev));
  return ADDS_OK;
}

static bool is_device_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

/* graph validation + weight canonicalisation, on the device */
__global__ void k_pack_edges(const uint32_t *dst, const uint32_t *w, uint64_t m, uint32_t n,
                             int is_float, uint2 *edges, unsigned *bad) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = dst[i];
    uint32_t x = w ? w[i] : 0u;
    if (d >= n) atomicOr(bad, 1u);
    if (is_float) {
      if (x == 0x80000000u) x = 0u; /* -0.0 -> +0.0: identical sums */
      if (x > 0x7F800000u) atomicOr(bad, 2u); /* negative or NaN */
    } else if (x > 0x7FFFFFFFu) {
      atomicOr(bad, 4u); /* negative as int32 */
    }
    edges[i] = make_uint2(d, x);
  }
}
__global__ void k_set_weights(uint2 *edges, const uint32_t *w, uint64_t m, int is_float,
                              unsigned *bad) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t x = w[i];
    if (is_float) {
      if (x == 0x80000000u) x = 0u;
      if (x > 0x7F800000u) atomicOr(bad, 2u);
    } else if (x > 0x7FFFFFFFu) {
      atomicOr(bad, 4u);
    }
    edges[i].y = x;
  }
}
/* New weights of several graphs in one launch, a CTA per SW_TILE edges: stored
 * and checked as k_set_weights does, and the sample that k_sample_w takes
 * summed where its edges lie in the tile. */
struct SwJob {
  uint2 *edges;
  const uint32_t *w;
  unsigned long long m;
  double sum;
  unsigned ns, tile0, is_float, bad;
};
constexpr unsigned SW_TILE = 4096;
__global__ void k_set_weights_many(SwJob *jobs, unsigned njobs) {
  unsigned lo = 0, hi = njobs - 1u;
  while (lo < hi) {
    const unsigned mid = (lo + hi + 1u) >> 1;
    if (jobs[mid].tile0 <= blockIdx.x) lo = mid; else hi = mid - 1u;
  }
  SwJob &J = jobs[lo];
  const uint64_t m = J.m, e0 = (uint64_t)(blockIdx.x - J.tile0) * SW_TILE;
  const uint64_t e1 = e0 + SW_TILE < m ? e0 + SW_TILE : m;
  const uint32_t *w = J.w;
  unsigned bad = 0;
  for (uint64_t i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
    uint32_t x = w[i];
    if (J.is_float) {
      if (x == 0x80000000u) x = 0u;
      if (x > 0x7F800000u) bad |= 2u;
    } else if (x > 0x7FFFFFFFu) {
      bad |= 4u;
    }
    J.edges[i].y = x;
  }
  double acc = 0;
  const unsigned ns = J.ns;
  const uint64_t s0 = (uint64_t)((double)e0 * ns / (double)m), s1 = (uint64_t)((double)e1 * ns / (double)m) + 2u;
  for (uint64_t i = (s0 > 2u ? s0 - 2u : 0u) + threadIdx.x; i < s1 && i < ns; i += blockDim.x) {
    uint64_t e = (uint64_t)((double)i * (double)m / (double)ns);
    if (e >= m) e = m - 1;
    if (e < e0 || e >= e1) continue;
    const uint32_t x = w[e];
    acc += J.is_float ? (x == 0x80000000u ? 0.0 : (double)__uint_as_float(x)) : (double)x;
  }
  bad = __reduce_or_sync(0xFFFFFFFFu, bad);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31u) == 0u) {
    if (bad) atomicOr(&J.bad, bad);
    if (acc != 0.0) atomicAdd(&J.sum, acc);
  }
}
__global__ void k_check_rows(const unsigned *row, uint32_t n, uint64_t m, unsigned *bad,
                             unsigned *maxdeg) {
  unsigned md = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const unsigned a = row[v], b = row[v + 1];
    if (b < a || b > m || (v == 0 && a != 0u) || (v == n - 1 && b != m)) atomicOr(bad, 8u);
    else md = max(md, b - a);
  }
  for (int o = 16; o > 0; o >>= 1) md = max(md, __shfl_down_sync(0xFFFFFFFFu, md, o));
  if ((threadIdx.x & 31u) == 0u) atomicMax(maxdeg, md);
}
/* .gr row end offsets (u64) -> u32 row[i0 + 1 + i]; an offset above m (it
 * would not fit the u32 CSR) is flagged, the order is checked later by
 * k_check_rows */
__global__ void k_rows_u64(const unsigned long long *ends, uint64_t cnt, uint64_t i0, uint64_t m,
                           unsigned *row, unsigned *bad) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned long long e = ends[i];
    if (e > m) atomicOr(bad, 8u);
    row[i0 + 1 + i] = (unsigned)(e > m ? m : e);
  }
}
/* evenly spaced weight sample (profiler_kernel, ads_int/kernel.cu:153-183) */
__global__ void k_sample_w(const uint2 *edges, uint64_t m, int is_float, unsigned ns, double *out) {
  double acc = 0;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += gridDim.x * blockDim.x) {
    const uint64_t e = (uint64_t)((double)i * (double)m / (double)ns);
    const uint32_t x = edges[e < m ? e : m - 1].y;
    acc += is_float ? (double)__uint_as_float(x) : (double)x;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31u) == 0u) atomicAdd(out, acc);
}

static int graph_finish(adds_graph *g) {
  /* checks, degree/weight statistics, streams, result buffer */
  unsigned *scratch = nullptr;
  CK(cudaMalloc(&scratch, 64));
  CK(cudaMemsetAsync(scratch, 0, 64, g->stream));
  k_check_rows<<<592, 256, 0, g->stream>>>(g->row, g->n, g->m, scratch, scratch + 1);
  const unsigned ns = (unsigned)std::min<uint64_t>(g->m, 1u << 16);
  if (ns) k_sample_w<<<64, 256, 0, g->stream>>>(g->edges, g->m, g->wt == ADDS_F32, ns, (double *)(scratch + 2));
  unsigned h[2];
  double sw = 0;
  CK(cudaMemcpyAsync(h, scratch, 8, cudaMemcpyDeviceToHost, g->stream));
  CK(cudaMemcpyAsync(&sw, scratch + 2, 8, cudaMemcpyDeviceToHost, g->stream));
  CK(cudaStreamSynchronize(g->stream));
  cudaFree(scratch);
  if (h[0]) return ADDS_ERR_FORMAT;
  g->max_deg = h[1];
  g->avg_deg = g->n ? (double)g->m / g->n : 0.0;
  g->avg_w = ns ? sw / ns : 1.0;
  CK(cudaMalloc(&g->dist, ((size_t)g->n ? g->n : 1) * 4));
  g->bytes += (size_t)g->n * 4;
  CK(cudaEventCreate(&g->ev0));
  CK(cudaEventCreate(&g->ev1));
  return ADDS_OK;
}

static adds_graph *graph_new(int device, adds_wtype wt) {
  adds_graph *g = new adds_graph();
  g->device = device;
  g->wt = wt;
  adds_opts_init(&g->tuned_opts);
  adds_opts_init(&g->tuned_wave);
  if (cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    delete g;
    return nullptr;
  }
  return g;
}

extern "C" void adds_graph_free(adds_graph *g) {
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  engine_free(g->eng);
  ph_engine_free(g->peng);
  wv_engine_free(g->weng);
  if (g->row) cudaFree(g->row);
  if (g->edges) cudaFree(g->edges);
  if (g->dist) cudaFree(g->dist);
  if (g->sedges) cudaFree(g->sedges);
  if (g->split.at) cudaFree(g->split.at);
  if (g->trow) cudaFree(g->trow);
  if (g->tedges) cudaFree(g->tedges);
  if (g->wfirst) cudaFree(g->wfirst);
  if (g->wpiece) cudaFree(g->wpiece);
  if (g->aux) cudaFree(g->aux);
  if (g->sw_jobs) cudaFree(g->sw_jobs);
  if (g->sort_buf) cudaFree(g->sort_buf);
  if (g->sort_tmp) cudaFree(g->sort_tmp);
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (g->cstream) cudaStreamSynchronize(g->cstream);
  if (g->stage) cudaFree(g->stage);
  for (int j = 0; j < 2; ++j) {
    if (g->ev_free[j]) cudaEventDestroy(g->ev_free[j]);
    if (g->ev_ready[j]) cudaEventDestroy(g->ev_ready[j]);
  }
  if (g->cstream) cudaStreamDestroy(g->cstream);
  for (int i = 0; i < adds_graph::kRing; ++i)
    for (int j = 0; j < 4; ++j)
      if (g->ring[i][j]) cudaEventDestroy(g->ring[i][j]);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
}

/* Uploads dst/w (host or device) + u32 rows into g; validates on device. */
static int graph_upload(adds_graph *g, const unsigned *row_host_u32, const uint32_t *dst,
                        const void *w) {
  const size_t m = g->m;
  CK(cudaMalloc(&g->row, ((size_t)g->n + 1) * 4));
  CK(cudaMalloc(&g->edges, (m + ADDS_EDGE_PAD) * sizeof(uint2)));
  g->bytes = ((size_t)g->n + 1) * 4 + m * sizeof(uint2);
  CK(cudaMemcpyAsync(g->row, row_host_u32, ((size_t)g->n + 1) * 4, cudaMemcpyHostToDevice, g->stream));
  /* stream dst/w through device staging buffers in chunks */
  const size_t CH = (size_t)1 << 26;
  uint32_t *sd = nullptr, *sw = nullptr;
  unsigned *bad = nullptr;
  const size_t chunk = std::min(m ? m : 1, CH);
  CK(cudaMalloc(&sd, chunk * 4));
  CK(cudaMalloc(&sw, chunk * 4));
  CK(cudaMalloc(&bad, 4));
  CK(cudaMemsetAsync(bad, 0, 4, g->stream));
  const bool dd = dst && is_device_ptr(dst), dw = w && is_device_ptr(w);
  for (size_t off = 0; off < m; off += CH) {
    const size_t c = std::min(CH, m - off);
    CK(cudaMemcpyAsync(sd, dst + off, c * 4, dd ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, g->stream));
    if (w)
      CK(cudaMemcpyAsync(sw, (const uint32_t *)w + off, c * 4,
                         dw ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, g->stream));
    k_pack_edges<<<592, 256, 0, g->stream>>>(sd, w ? sw : nullptr, c, g->n, g->wt == ADDS_F32,
                                             g->edges + off, bad);
    /* the staging buffers are reused: wait before the next chunk */
    CK(cudaStreamSynchronize(g->stream));
  }
  unsigned hb = 0;
  CK(cudaMemcpyAsync(&hb, bad, 4, cudaMemcpyDeviceToHost, g->stream));
  CK(cudaStreamSynchronize(g->stream));
  cudaFree(sd);
  cudaFree(sw);
  cudaFree(bad);
  if (hb & 1u) return ADDS_ERR_FORMAT;
  if (hb & 6u) return ADDS_ERR_INVALID;
  return graph_finish(g);
}

/* ------------------------------------------------------------------------ */
/* Host -> device ingest through pinned staging.  Replaces the per-edge host
 * loop of readFromGR (ads_int/csr_graph.cu:260-280) and the pageable
 * cudaMemcpy calls of copy_to_gpu (csr_graph.cu:309-328): several host
 * threads read the next piece (pread from the file, or memcpy from caller
 * memory) into one of two pinned buffers while the GPU copies the other
 * piece in and converts it (row offsets u64 -> u32, {dst, weight} packing
 * and checks).  Nothing is parsed on the host. */
struct HostSrc {
  int fd = -1;                 /* pread from this file at off + byte offset ... */
  uint64_t off = 0;
  const char *mem = nullptr;   /* ... or copy from this address                */
  bool present() const { return fd >= 0 || mem != nullptr; }
};

static bool host_fill(const HostSrc &s, void *out, uint64_t at, size_t bytes, int nth) {
  if (bytes == 0) return true;
  const size_t min_slice = (size_t)1 << 20;
  int t = (int)std::min<size_t>((size_t)nth, (bytes + min_slice - 1) / min_slice);
  if (t < 1) t = 1;
  std::vector<char> ok((size_t)t, 1);
  auto part = [&](int i) {
    const size_t a = bytes * (size_t)i / (size_t)t, b = bytes * (size_t)(i + 1) / (size_t)t;
    char *o = (char *)out + a;
    if (s.mem) {
      memcpy(o, s.mem + at + a, b - a);
      return;
    }
    size_t done = 0;
    while (done < b - a) {
      const ssize_t r = pread(s.fd, o + done, b - a - done, (off_t)(s.off + at + a + done));
      if (r <= 0) {
        if (r < 0 && errno == EINTR) continue;
        ok[(size_t)i] = 0;
        return;
      }
      done += (size_t)r;
    }
  };
  std::vector<std::thread> th;
  for (int i = 1; i < t; ++i) th.emplace_back(part, i);
  part(0);
  for (auto &x : th) x.join();
  for (char c : ok)
    if (!c) return false;
  return true;
}

/* rows: the n row END offsets as u64 (row[0] = 0 is implied); dst and w:
 * m u32 words each (w absent = all-zero weights, as a .gr without edge
 * data).  g->n and g->m are set.  Ends with graph_finish's checks. */
static int graph_ingest(adds_graph *g, const HostSrc &rows, const HostSrc &dst, const HostSrc &w) {
  const uint64_t n = g->n, m = g->m;
  constexpr uint64_t CH = (uint64_t)1 << 22; /* words per piece: 16 MB of dst + 16 MB of w */
  constexpr size_t BUF = (size_t)CH * 8;     /* bytes per staging buffer                   */
  const int nth = (int)std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
  CK(cudaMalloc(&g->row, (n + 1) * 4));
  CK(cudaMalloc(&g->edges, (m + ADDS_EDGE_PAD) * sizeof(uint2)));
  g->bytes = (n + 1) * 4 + m * sizeof(uint2);
  CK(cudaMemsetAsync(g->row, 0, 4, g->stream));
  CK(cudaMemsetAsync(g->edges + m, 0, ADDS_EDGE_PAD * sizeof(uint2), g->stream));
  char *pin[2] = {nullptr, nullptr};
  char *dev = nullptr;
  unsigned *bad = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  int rc = ADDS_OK;
  auto cu = [&](cudaError_t e, const char *what) {
    if (e != cudaSuccess && rc == ADDS_OK) rc = cuda_fail(e, what);
    return rc == ADDS_OK;
  };
  if (cu(cudaHostAlloc((void **)&pin[0], BUF, cudaHostAllocDefault), "pinned staging") &&
      cu(cudaHostAlloc((void **)&pin[1], BUF, cudaHostAllocDefault), "pinned staging") &&
      cu(cudaMalloc(&dev, 2 * BUF), "device staging") && cu(cudaMalloc(&bad, 4), "flag") &&
      cu(cudaMemsetAsync(bad, 0, 4, g->stream), "flag") &&
      cu(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming), "event") &&
      cu(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming), "event")) {
    /* pieces: row ends in CH-entry pieces, then edges in CH-edge pieces */
    const uint64_t nrp = (n + CH - 1) / CH, nep = (m + CH - 1) / CH;
    for (uint64_t c = 0; c < nrp + nep && rc == ADDS_OK; ++c) {
      const int k = (int)(c & 1);
      if (c >= 2 && !cu(cudaEventSynchronize(ev[k]), "staging wait")) break;
      char *p = pin[k], *d = dev + (size_t)k * BUF;
      if (c < nrp) {
        const uint64_t i0 = c * CH, cnt = std::min(CH, n - i0);
        if (!host_fill(rows, p, i0 * 8, cnt * 8, nth)) {
          rc = ADDS_ERR_IO;
          break;
        }
        if (!cu(cudaMemcpyAsync(d, p, cnt * 8, cudaMemcpyHostToDevice, g->stream), "rows H2D") ||
            !cu(cudaEventRecord(ev[k], g->stream), "event"))
          break;
        k_rows_u64<<<592, 256, 0, g->stream>>>((const unsigned long long *)d, cnt, i0, m, g->row,
                                              bad);
      } else {
        const uint64_t i0 = (c - nrp) * CH, cnt = std::min(CH, m - i0);
        if (!host_fill(dst, p, i0 * 4, cnt * 4, nth) ||
            (w.present() && !host_fill(w, p + CH * 4, i0 * 4, cnt * 4, nth))) {
          rc = ADDS_ERR_IO;
          break;
        }
        if (!cu(cudaMemcpyAsync(d, p, cnt * 4, cudaMemcpyHostToDevice, g->stream), "dst H2D") ||
            (w.present() && !cu(cudaMemcpyAsync(d + CH * 4, p + CH * 4, cnt * 4,
                                                cudaMemcpyHostToDevice, g->stream), "w H2D")) ||
            !cu(cudaEventRecord(ev[k], g->stream), "event"))
          break;
        k_pack_edges<<<592, 256, 0, g->stream>>>((const uint32_t *)d,
                                                w.present() ? (const uint32_t *)(d + CH * 4)
                                                            : nullptr,
                                                cnt, (uint32_t)n, g->wt == ADDS_F32,
                                                g->edges + i0, bad);
      }
      cu(cudaGetLastError(), "convert kernel");
    }
  }
  unsigned hb = 0;
  if (rc == ADDS_OK) {
    cu(cudaMemcpyAsync(&hb, bad, 4, cudaMemcpyDeviceToHost, g->stream), "flag D2H");
    cu(cudaStreamSynchronize(g->stream), "ingest");
  } else {
    cudaStreamSynchronize(g->stream);
  }
  for (int k = 0; k < 2; ++k) {
    if (ev[k]) cudaEventDestroy(ev[k]);
    if (pin[k]) cudaFreeHost(pin[k]);
  }
  if (dev) cudaFree(dev);
  if (bad) cudaFree(bad);
  if (rc) return rc;
  if (hb & 9u) return ADDS_ERR_FORMAT; /* dst >= n, row offset > m */
  if (hb & 6u) return ADDS_ERR_INVALID; /* negative or NaN weight */
  return graph_finish(g);
}

extern "C" int adds_graph_from_csr(uint32_t n, uint64_t m, const uint64_t *row_start,
                                   const uint32_t *dst, const void *w, adds_wtype wt, int device,
                                   adds_graph **out) {
  if (!out || !row_start || (m && !dst) || n == 0 || n >= 0x80000000u || m >= 0xFFFFFFFFull ||
      (wt != ADDS_I32 && wt != ADDS_F32))
    return ADDS_ERR_INVALID;
  *out = nullptr;
  int rc = set_device(device);
  if (rc) return rc;
  if (row_start[0] != 0 || row_start[n] != m) return ADDS_ERR_INVALID;
  const bool dev_arrays = (dst && is_device_ptr(dst)) || (w && is_device_ptr(w));
  adds_graph *g = graph_new(device, wt);
  if (!g) return ADDS_ERR_CUDA;
  g->n = n;
  g->m = m;
  if (!dev_arrays) {
    /* host arrays: pinned, pipelined upload; the rows are checked on the GPU */
    HostSrc rs, ds, ws;
    rs.mem = (const char *)(row_start + 1);
    ds.mem = (const char *)dst;
    ws.mem = (const char *)w;
    rc = graph_ingest(g, rs, ds, ws);
  } else {
    std::vector<unsigned> row(n + 1);
    for (uint32_t v = 0; v <= n && !rc; ++v) {
      if (v && row_start[v] < row_start[v - 1]) rc = ADDS_ERR_INVALID;
      row[v] = (unsigned)row_start[v];
    }
    if (!rc) rc = graph_upload(g, row.data(), dst, w);
  }
  if (rc) {
    adds_graph_free(g);
    return rc;
  }
  *out = g;
  return ADDS_OK;
}

/* .gr v1 reader (readFromGR, ads_int/csr_graph.cu:203-296): the header and
 * the file size are checked on the host; out_end[], dst[] and w[] are read
 * by host threads straight into pinned staging buffers and converted and
 * checked on the GPU (graph_ingest). */
extern "C" int adds_graph_load_gr(const char *path, adds_wtype wt, int device, adds_graph **out) {
  if (!path || !out || (wt != ADDS_I32 && wt != ADDS_F32)) return ADDS_ERR_INVALID;
  *out = nullptr;
  int rc = set_device(device);
  if (rc) return rc;
  const int fd = open(path, O_RDONLY);
  if (fd < 0) return ADDS_ERR_IO;
  struct stat sb;
  uint64_t h[4];
  if (fstat(fd, &sb) != 0) {
    close(fd);
    return ADDS_ERR_IO;
  }
  const size_t len = (size_t)sb.st_size;
  if (len < 32 || pread(fd, h, 32, 0) != 32) {
    close(fd);
    return len < 32 ? ADDS_ERR_FORMAT : ADDS_ERR_IO;
  }
  const uint64_t version = h[0], esz = h[1], n64 = h[2], m64 = h[3];
  rc = ADDS_OK;
  adds_graph *g = nullptr;
  if (version != 1 || (esz != 0 && esz != 4) || n64 == 0 || n64 >= 0x80000000ull ||
      m64 >= 0xFFFFFFFFull) {
    rc = ADDS_ERR_FORMAT;
  } else {
    const size_t need = 32 + 8 * n64 + 4 * m64 + ((m64 & 1) ? 4 : 0) + (esz ? 4 * m64 : 0);
    if (len < need) rc = ADDS_ERR_FORMAT;
  }
  if (!rc) {
    g = graph_new(device, wt);
    if (!g) rc = ADDS_ERR_CUDA;
    else {
      g->n = (uint32_t)n64;
      g->m = m64;
      HostSrc rs, ds, ws;
      rs.fd = ds.fd = fd;
      rs.off = 32;
      ds.off = 32 + 8 * n64;
      if (esz) {
        ws.fd = fd;
        ws.off = ds.off + 4 * m64 + ((m64 & 1) ? 4 : 0);
      }
      rc = graph_ingest(g, rs, ds, ws);
    }
  }
  close(fd);
  if (rc) {
    if (g) adds_graph_free(g);
    return rc;
  }
  *out = g;
  return ADDS_OK;
}

extern "C" int adds_graph_generate(const adds_gen_spec *spec, int device, adds_graph **out) {
  if (!spec || !out) return ADDS_ERR_INVALID;
  *out = nullptr;
  int rc = set_device(device);
  if (rc) return rc;
  adds_graph *g = graph_new(device, spec->wtype);
  if (!g) return ADDS_ERR_CUDA;
  uint32_t n = 0;
  uint64_t m = 0;
  rc = adds_gen_build(spec, &g->row, &g->edges, &n, &m, g->stream);
  if (!rc) {
    g->n = n;
    g->m = m;
    g->bytes = ((size_t)n + 1) * 4 + m * sizeof(uint2);
    rc = graph_finish(g);
  }
  if (rc) {
    adds_graph_free(g);
    return rc;
  }
  *out = g;
  return ADDS_OK;
}

extern "C" int adds_graph_info(const adds_graph *g, adds_graph_info_t *info) {
  if (!g || !info) return ADDS_ERR_INVALID;
  info->n = g->n;
  info->m = g->m;
  info->wtype = g->wt;
  info->device = g->device;
  info->max_degree = g->max_deg;
  info->avg_degree = g->avg_deg;
  info->avg_weight = g->avg_w;
  info->device_bytes = g->bytes + g->eng.bytes + g->peng.bytes + g->weng.bytes +
                       (g->sort_buf ? (size_t)g->m * 16 : 0) + g->sort_tmp_bytes +
                       g->sw_cap * sizeof(SwJob);
  return ADDS_OK;
}

extern "C" int adds_graph_download(const adds_graph *g, uint64_t *row_start, uint32_t *dst, void *w) {
  if (!g) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(g->device));
  if (row_start) {
    std::vector<unsigned> r(g->n + 1);
    CK(cudaMemcpy(r.data(), g->row, ((size_t)g->n + 1) * 4, cudaMemcpyDeviceToHost));
    for (size_t i = 0; i <= g->n; ++i) row_start[i] = r[i];
  }
  if (dst || w) {
    const size_t CH = (size_t)1 << 24;
    std::vector<uint2> buf(std::min<size_t>(g->m ? g->m : 1, CH));
    for (size_t off = 0; off < g->m; off += CH) {
      const size_t c = std::min(CH, (size_t)g->m - off);
      CK(cudaMemcpy(buf.data(), g->edges + off, c * sizeof(uint2), cudaMemcpyDeviceToHost));
      for (size_t i = 0; i < c; ++i) {
        if (dst) dst[off + i] = buf[i].x;
        if (w) ((uint32_t *)w)[off + i] = buf[i].y;
      }
    }
  }
  return ADDS_OK;
}

extern "C" int adds_graph_set_weights(adds_graph *g, const void *w) {
  if (!g || !w) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(g->device));
  if (g->m == 0) return ADDS_OK;
  const uint32_t *src = (const uint32_t *)w;
  uint32_t *tmp = nullptr;
  if (!is_device_ptr(w)) {
    CK(cudaMalloc(&tmp, g->m * 4));
    CK(cudaMemcpyAsync(tmp, w, g->m * 4, cudaMemcpyHostToDevice, g->stream));
    src = tmp;
  }
  if (!g->aux) CK(cudaMalloc(&g->aux, 64));
  CK(cudaMemsetAsync(g->aux, 0, 64, g->stream));
  k_set_weights<<<592, 256, 0, g->stream>>>(g->edges, src, g->m, g->wt == ADDS_F32, g->aux);
  /* the weight sample feeds the automatic delta */
  const unsigned ns = (unsigned)std::min<uint64_t>(g->m, 1u << 16);
  k_sample_w<<<64, 256, 0, g->stream>>>(g->edges, g->m, g->wt == ADDS_F32, ns,
                                         (double *)(g->aux + 2));
  unsigned h[4] = {0, 0, 0, 0};
  CK(cudaMemcpyAsync(h, g->aux, 16, cudaMemcpyDeviceToHost, g->stream));
  CK(cudaStreamSynchronize(g->stream));
  if (tmp) cudaFree(tmp);
  if (h[0]) return ADDS_ERR_INVALID;
  double sw;
  memcpy(&sw, h + 2, 8);
  g->avg_w = sw / ns;
  g->sorted_valid = false; /* the weight order changed */
  g->trans_valid = false;  /* the in-edges carry weights */
  ++g->wversion;
  return ADDS_OK;
}

/* One launch and one wait for all of them: one by one each costs a clear, two
 * launches, a copy back and a wait, 33 us, which the work of a graph of 65,536
 * vertices does not fill (a training step on 128 of them: 26.4 ms so, 21.8 ms
 * together). */
extern "C" int adds_graphs_set_weights(adds_graph *const *graphs, const void *const *w, uint32_t ng) {
  if (ng && (!graphs || !w)) return ADDS_ERR_INVALID;
  bool together = ng > 1;
  for (uint32_t i = 0; i < ng; ++i) {
    if (!graphs[i] || !w[i]) return ADDS_ERR_INVALID;
    /* one by one: host arrays, several devices, a graph named twice */
    if (graphs[i]->device != graphs[0]->device || !is_device_ptr(w[i])) together = false;
  }
  if (together) {
    std::vector<adds_graph *> named(graphs, graphs + ng);
    std::sort(named.begin(), named.end());
    together = std::adjacent_find(named.begin(), named.end()) == named.end();
  }
  if (!together) {
    for (uint32_t i = 0; i < ng; ++i) {
      const int rc = adds_graph_set_weights(graphs[i], w[i]);
      if (rc) return rc;
    }
    return ADDS_OK;
  }
  adds_graph *g0 = graphs[0];
  CK(cudaSetDevice(g0->device));
  std::vector<SwJob> jobs;
  unsigned long long tiles = 0;
  for (uint32_t i = 0; i < ng; ++i) {
    adds_graph *g = graphs[i];
    CK(cudaStreamSynchronize(g->stream)); /* solves that read the old weights */
    SwJob j;
    j.edges = g->edges;
    j.w = (const uint32_t *)w[i];
    j.m = g->m;
    j.sum = 0;
    j.ns = (unsigned)std::min<uint64_t>(g->m, 1u << 16);
    j.tile0 = (unsigned)tiles;
    j.is_float = g->wt == ADDS_F32;
    j.bad = 0;
    if (g->m == 0) continue;
    tiles += (g->m + SW_TILE - 1) / SW_TILE;
    jobs.push_back(j);
  }
  if (jobs.empty()) return ADDS_OK;
  if (tiles > 0x7FFFFFFFull) return ADDS_ERR_UNSUPPORTED;
  if (g0->sw_cap < jobs.size()) {
    if (g0->sw_jobs) cudaFree(g0->sw_jobs);
    g0->sw_jobs = nullptr;
    g0->sw_cap = 0;
    CK(cudaMalloc(&g0->sw_jobs, jobs.size() * sizeof(SwJob)));
    g0->sw_cap = jobs.size();
  }
  SwJob *d = (SwJob *)g0->sw_jobs;
  CK(cudaMemcpyAsync(d, jobs.data(), jobs.size() * sizeof(SwJob), cudaMemcpyHostToDevice, g0->stream));
  k_set_weights_many<<<(unsigned)tiles, 256, 0, g0->stream>>>(d, (unsigned)jobs.size());
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(jobs.data(), d, jobs.size() * sizeof(SwJob), cudaMemcpyDeviceToHost, g0->stream));
  CK(cudaStreamSynchronize(g0->stream));
  int rc = ADDS_OK;
  for (uint32_t i = 0, k = 0; i < ng; ++i) {
    adds_graph *g = graphs[i];
    if (g->m == 0) continue;
    const SwJob &j = jobs[k++];
    if (j.bad) {
      rc = ADDS_ERR_INVALID;
      continue;
    }
    g->avg_w = j.sum / j.ns;
    g->sorted_valid = false;
    g->trans_valid = false;
    ++g->wversion;
  }
  return rc;
}

extern "C" int adds_graph_save_gr(const adds_graph *g, const char *path) {
  if (!g || !path) return ADDS_ERR_INVALID;
  std::vector<uint64_t> row(g->n + 1);
  std::vector<uint32_t> dst(g->m), w(g->m);
  int rc = adds_graph_download(g, row.data(), dst.data(), w.data());
  if (rc) return rc;
  FILE *f = fopen(path, "wb");
  if (!f) return ADDS_ERR_IO;
  const uint64_t hdr[4] = {1, 4, g->n, g->m};
  bool ok = fwrite(hdr, 8, 4, f) == 4;
  ok = ok && fwrite(row.data() + 1, 8, g->n, f) == g->n;
  ok = ok && fwrite(dst.data(), 4, g->m, f) == g->m;
  if (g->m & 1) {
    const uint32_t pad = 0;
    ok = ok && fwrite(&pad, 4, 1, f) == 1;
  }
  ok = ok && fwrite(w.data(), 4, g->m, f) == g->m;
  if (fclose(f) != 0) ok = false;
  return ok ? ADDS_OK : ADDS_ERR_IO;
}

/* ------------------------------------------------------------------------ */
/* knob resolution: explicit opts > tuned values > degree/weight heuristic   */
static float auto_scale(const adds_graph *g) {
  const double aw = g->avg_w > 1e-30 ? g->avg_w : 1.0;
  return (float)(65536.0 / aw); /* 1 key unit = avg_w / 2^16 */
}

/* Delta ~ 4 * avg_weight / avg_degree (the reference starts from
 * avg_wt/avg_degree/32 and raises it on the device, wl.h:414-440, 968-1360;
 * on 148 SMs a wider bucket is the better starting point: measured best for
 * R-MAT 22/24 at 4x). */
static int auto_shift(const adds_graph *g) {
  const double deg = g->avg_deg > 1.0 ? g->avg_deg : 1.0;
  double delta_keys;
  if (g->wt == ADDS_F32) delta_keys = 4.0 * 65536.0 / deg;
  else delta_keys = 4.0 * (g->avg_w > 1.0 ? g->avg_w : 1.0) / deg;
  int s = (int)lround(log2(delta_keys > 1.0 ? delta_keys : 1.0));
  return std::max(0, std::min(s, 31));
}

/* The knobs of a solve on g: the caller's, else g's tuned ones (unless
 * use_tuned is false), else the defaults.  The tuned ones are an engine's: a
 * wave kernel takes none of them. */
static void resolve(const adds_graph *g, const adds_opts *o, Knobs *k, int *shift, float *scale,
                    bool use_tuned = true) {
  adds_opts d;
  adds_opts_init(&d);
  if (!o) o = &d;
  const bool wave = o->wave > 0 && !g->wave_off;
  const adds_opts *t = (g->tuned && use_tuned && !wave) ? &g->tuned_opts : &d;
  *shift = o->delta_shift >= 0 ? o->delta_shift : (t->delta_shift >= 0 ? t->delta_shift : auto_shift(g));
  *scale = o->delta_scale > 0 ? o->delta_scale : (t->delta_scale > 0 ? t->delta_scale : auto_scale(g));
  k->window = o->window > 0 ? o->window : (t->window > 0 ? t->window : 2);
  k->ctas_per_sm = o->ctas_per_sm > 0 ? o->ctas_per_sm : t->ctas_per_sm;
  k->batch_max = o->batch_max > 0 ? o->batch_max : (t->batch_max > 0 ? t->batch_max : 512);

  k->strict = o->strict_order >= 0 ? o->strict_order : (t->strict_order >= 0 ? t->strict_order : 1);
  k->local_max = o->local_max >= 0 ? o->local_max : (t->local_max >= 0 ? t->local_max : 512);
  k->near_far = (o->near_far > 0 || t->near_far > 0) ? 1 : 0;
  k->block = o->block_threads > 0 ? o->block_threads : (t->block_threads > 0 ? t->block_threads : 256);
  k->greed = o->greed >= 0 ? o->greed : (t->greed >= 0 ? t->greed : 4);
  k->engine = o->engine > 0 ? o->engine : (t->engine > 0 ? t->engine : ADDS_ENGINE_PHASE);
  if (k->engine != ADDS_ENGINE_ASYNC) k->engine = ADDS_ENGINE_PHASE;
  /* light/heavy split: adaptive (2) in the phase engine, always (1) in the
   * asynchronous one, which treats 2 as 1 */
  k->light_heavy = o->light_heavy >= 0 ? o->light_heavy
                                       : (t->light_heavy >= 0 ? t->light_heavy
                                                              : (k->engine == ADDS_ENGINE_PHASE ? 2 : 1));
  /* on-device bucket width: on in the asynchronous engine (its window on
   * the 4096^2 grid: 20.8-23.5 ms from bucket shift 17 to 19 against
   * 21.6-44.4 ms fixed), off in the phase engine unless asked or tuned */
  k->adapt = o->adapt >= 0 ? o->adapt
                           : (t->adapt >= 0 ? t->adapt : (k->engine == ADDS_ENGINE_ASYNC ? 1 : 0));
  const int hub_def = k->engine == ADDS_ENGINE_PHASE ? 256 : 16384;
  k->hub_threshold = o->hub_threshold > 0 ? o->hub_threshold : (t->hub_threshold > 0 ? t->hub_threshold : hub_def);
  k->hub_chunk = 4096;
  if (k->engine == ADDS_ENGINE_PHASE) {
    const int pb = o->block_threads > 0 ? o->block_threads : (t->block_threads > 0 ? t->block_threads : 256);
    const int pc = o->ctas_per_sm > 0 ? o->ctas_per_sm : (t->ctas_per_sm > 0 ? t->ctas_per_sm : 4);
    k->variant = phase_variant(pb, pc);
  } else {
    k->variant = 0;
  }
  k->group_ctas = o->group_ctas > 0 ? o->group_ctas : (t->group_ctas > 0 ? t->group_ctas : 0);
  k->solo_max = o->solo_max >= 0 ? o->solo_max : (t->solo_max >= 0 ? t->solo_max : 1024);
  /* dense bucket slots: explicit > tuned > off (measured on R-MAT 24: the
   * scans remove the stale entries but cost as much as they save) */
  k->dense_scan = o->dense_scan != 0 ? o->dense_scan : (t->dense_scan != 0 ? t->dense_scan : -1);
  /* pull heavy phases: 1 asked for, 0 off, 2 automatic (graphs of at least
   * 2^22 edges; the leader still picks push wherever the counted pull would
   * read more edges) */
  k->pull = o->pull != 0 ? (o->pull > 0 ? 1 : 0) : (t->pull != 0 ? (t->pull > 0 ? 1 : 0) : 2);
  const int tmo = o->timeout_ms > 0 ? o->timeout_ms : 20000;
  k->timeout_ns = (unsigned long long)tmo * 1000000ull;
  k->wave = o->wave > 0 ? std::min(o->wave - 1, WV_LAST) : -1;
}

/* True when the caller leaves the choice of engine and schedule to the
 * library: only then may a solve go to the wave kernels by itself. */
static bool schedule_auto(const adds_opts *o) {
  return !o || (o->engine <= 0 && o->wave == 0 && o->delta_shift < 0 && o->delta_scale <= 0.f &&
                o->window <= 0 && o->ctas_per_sm <= 0 && o->batch_max <= 0 &&
                o->hub_threshold <= 0 && o->adapt < 0 && o->strict_order < 0 &&
                o->local_max < 0 && o->light_heavy < 0 && o->block_threads <= 0 &&
                o->greed < 0 && o->group_ctas <= 0 && o->solo_max < 0 && o->near_far <= 0 &&
                o->dense_scan == 0 && o->pull == 0);
}

/* ------------------------------------------------------------------------ */
/* light/heavy support: a copy of the CSR with each row sorted by weight and,
 * for the current bucket width, the number of light edges (w < delta) at the
 * start of each row.  Heavy edges cannot land in the bucket their tail
 * vertex is in, so they are relaxed once, after that bucket has settled. */
__global__ void k_unzip(const uint2 *e, uint64_t m, uint32_t *w, uint32_t *d) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 x = e[i];
    w[i] = x.y;
    d[i] = x.x;
  }
}
__global__ void k_zip(const uint32_t *w, const uint32_t *d, uint64_t m, uint2 *e) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    e[i] = make_uint2(d[i], w[i]);
}
__global__ void k_split(const unsigned *row, const uint2 *se, uint32_t n, unsigned thr,
                        unsigned *split) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    unsigned lo = row[v], hi = row[v + 1];
    const unsigned r0 = lo;
    while (lo < hi) { /* first edge with weight >= thr */
      const unsigned mid = lo + ((hi - lo) >> 1);
      if (se[mid].y < thr) lo = mid + 1; else hi = mid;
    }
    split[v] = lo - r0;
  }
}

static int graph_sorted(adds_graph *g) {
  if (g->sorted_valid) return ADDS_OK;
  const size_t m = g->m;
  if (!g->sedges) {
    CK(cudaMalloc(&g->sedges, (m + ADDS_EDGE_PAD) * sizeof(uint2)));
    CK(cudaMemsetAsync(g->sedges + m, 0, ADDS_EDGE_PAD * sizeof(uint2), g->stream));
    g->bytes += m * sizeof(uint2);
  }
  if (m == 0) {
    g->sorted_valid = true;
    return ADDS_OK;
  }
  if (m >= 0x7FFFFFFFull) return ADDS_ERR_UNSUPPORTED;
  if (!g->sort_buf) CK(cudaMalloc(&g->sort_buf, m * 16)); /* kept for re-sorts */
  uint32_t *wk = g->sort_buf, *dv = wk + m, *wk2 = wk + 2 * m, *dv2 = wk + 3 * m;
  k_unzip<<<592, 256, 0, g->stream>>>(g->edges, m, wk, dv);
  size_t tb = 0;
  cub::DeviceSegmentedSort::SortPairs(nullptr, tb, wk, wk2, dv, dv2, (int)m, (int)g->n, g->row,
                                      g->row + 1, g->stream);
  if (tb > g->sort_tmp_bytes) {
    if (g->sort_tmp) cudaFree(g->sort_tmp);
    g->sort_tmp = nullptr;
    g->sort_tmp_bytes = 0;
    CK(cudaMalloc(&g->sort_tmp, tb));
    g->sort_tmp_bytes = tb;
  }
  cudaError_t e = cub::DeviceSegmentedSort::SortPairs(g->sort_tmp, tb, wk, wk2, dv, dv2, (int)m,
                                                      (int)g->n, g->row, g->row + 1, g->stream);
  if (e == cudaSuccess) k_zip<<<592, 256, 0, g->stream>>>(wk2, dv2, m, g->sedges);
  if (e != cudaSuccess) return cuda_fail(e, "segmented sort");
  if (m > (1ull << 24)) {
    /* a large graph's sort buffers (16 B per edge, plus CUB's) are not kept:
     * weight updates that need a re-sort are rare there, and the memory is
     * better left to the solver */
    CK(cudaStreamSynchronize(g->stream));
    cudaFree(g->sort_buf);
    g->sort_buf = nullptr;
    cudaFree(g->sort_tmp);
    g->sort_tmp = nullptr;
    g->sort_tmp_bytes = 0;
  }
  g->sorted_valid = true;
  return ADDS_OK;
}

/* light threshold in weight bits for bucket width 2^shift key units */
static unsigned light_threshold(const adds_graph *g, int shift, float scale) {
  if (g->wt == ADDS_I32) return shift >= 31 ? 0xFFFFFFFFu : (1u << shift);
  const double dw = ldexp(1.0, shift) / (double)scale;
  if (!(dw < 3.0e38)) return 0xFFFFFFFFu;
  const float f = (float)dw;
  unsigned b;
  memcpy(&b, &f, 4);
  return b;
}

/* S for threshold thr and g's present weights.  *rebuilt: work was queued on
 * the graph's stream. */
static int graph_split(adds_graph *g, Split &S, unsigned thr, bool *rebuilt) {
  *rebuilt = !g->sorted_valid;
  int rc = graph_sorted(g);
  if (rc) return rc;
  if (S.valid && S.thr == thr && S.wversion == g->wversion) return ADDS_OK;
  *rebuilt = true;
  S.valid = false;
  if (!S.at) {
    CK(cudaMalloc(&S.at, ((size_t)g->n ? g->n : 1) * 4));
    if (&S == &g->split) g->bytes += (size_t)g->n * 4;
  }
  k_split<<<592, 256, 0, g->stream>>>(g->row, g->sedges, g->n, thr, S.at);
  CK(cudaGetLastError());
  S.thr = thr;
  S.wversion = g->wversion;
  S.valid = true;
  return ADDS_OK;
}

/* Edge array and light counts the engine should use for this graph; S belongs
 * to the caller (a plain solve or a batch). */
static int graph_layout(adds_graph *g, Split &S, const Knobs &k, int shift, float scale,
                        const uint2 **edges, const unsigned **split) {
  if (!k.light_heavy) {
    *edges = g->edges;
    *split = nullptr;
    return ADDS_OK;
  }
  bool rebuilt;
  const int rc = graph_split(g, S, light_threshold(g, shift, scale), &rebuilt);
  if (rc) return rc;
  /* the rebuild ran on the graph's stream; solves may run on another */
  if (rebuilt) CK(cudaStreamSynchronize(g->stream));
  *edges = g->sedges;
  *split = S.at;
  return ADDS_OK;
}

/* In-edge CSR for pull phases: in-degrees by atomic counts, their exclusive
 * scan, then each out-edge u -> v written as {u, w} at a cursor of v (the
 * order inside an in-row is whatever the atomics give; a pull takes the
 * minimum over the row, which does not depend on it).  A warp per tail
 * vertex reads its row coalesced. */
__global__ void k_indeg(const uint2 *e, uint64_t m, unsigned *cnt) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + e[i].x, 1u);
}
__global__ void k_transpose(const unsigned *row, const uint2 *e, uint32_t n, unsigned *cur,
                            uint2 *te) {
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t wstride = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t u = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; u < n; u += wstride) {
    const unsigned r1 = row[u + 1];
    for (unsigned i = row[u] + lane; i < r1; i += 32u) {
      const uint2 x = e[i];
      te[atomicAdd(cur + x.x, 1u)] = make_uint2((unsigned)u, x.y);
    }
  }
}

static int graph_transposed(adds_graph *g) {
  if (g->trans_valid) return ADDS_OK;
  const size_t n = g->n, m = g->m;
  if (!g->trow || !g->tedges) {
    if (g->trow) cudaFree(g->trow);
    g->trow = nullptr;
    CK(cudaMalloc(&g->trow, (n + 1) * 4));
    const cudaError_t ea = cudaMalloc(&g->tedges, (m + ADDS_EDGE_PAD) * sizeof(uint2));
    if (ea != cudaSuccess) {
      cudaFree(g->trow);
      g->trow = nullptr;
      g->tedges = nullptr;
      return cuda_fail(ea, "transposed graph");
    }
    CK(cudaMemsetAsync(g->tedges + m, 0, ADDS_EDGE_PAD * sizeof(uint2), g->stream));
    g->bytes += (n + 1) * 4 + m * sizeof(uint2);
  }
  unsigned *cnt = nullptr;
  void *tmp = nullptr;
  size_t tb = 0;
  int rc = ADDS_OK;
  cudaError_t e = cudaMalloc(&cnt, (n + 1) * 4);
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, (n + 1) * 4, g->stream);
  if (e == cudaSuccess && m) {
    k_indeg<<<4 * 148, 256, 0, g->stream>>>(g->edges, m, cnt);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, g->trow, (int)(n + 1), g->stream);
  if (e == cudaSuccess) e = cudaMalloc(&tmp, tb ? tb : 16);
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, g->trow, (int)(n + 1), g->stream);
  /* the cursors start at the row offsets */
  if (e == cudaSuccess) e = cudaMemcpyAsync(cnt, g->trow, n * 4, cudaMemcpyDeviceToDevice, g->stream);
  if (e == cudaSuccess && m) {
    k_transpose<<<4 * 148, 256, 0, g->stream>>>(g->row, g->edges, g->n, cnt, g->tedges);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) rc = cuda_fail(e, "transposed graph");
  if (cnt) cudaFree(cnt);
  if (tmp) cudaFree(tmp);
  if (!rc) g->trans_valid = true;
  return rc;
}

/* The in-edge CSR of q's graph when pull phases may run on it (phase engine,
 * light/heavy split, bucket ring; automatic: 2^22 edges or more, where a
 * heavy phase is long enough to pay for the extra launches of a pull); else
 * none. */
static int phase_pull_arrays(adds_graph *g, const Knobs &k, PhQuery *q) {
  q->trow = nullptr;
  q->tedges = nullptr;
  if (!k.pull || !q->split || k.near_far || g->m == 0) return ADDS_OK;
  if (k.pull == 2 && g->m < (1ull << 22)) return ADDS_OK;
  if (g->n >= 0x7FFFFFFFu || g->m >= 0xFFFFFFFFull) return ADDS_OK; /* 32-bit offsets */
  const int rc = graph_transposed(g);
  if (rc) return rc;
  q->trow = g->trow;
  q->tedges = g->tedges;
  return ADDS_OK;
}

/* ------------------------------------------------------------------------ */
/* plain solves                                                               */
static int graph_engine(adds_graph *g, const Knobs &k, int shift, float scale) {
  const uint2 *edges;
  const unsigned *split;
  int rc = graph_layout(g, g->split, k, shift, scale, &edges, &split);
  if (rc) return rc;
  if (g->eng.nq == 1) {
    QueryDesc &d = g->eng.qs_host[0];
    if (d.shift0 == (unsigned)shift && d.scale == scale && d.edges == edges && d.split == split)
      return ADDS_OK;
    /* same sizing: only the descriptor changes */
    d.shift0 = (unsigned)shift;
    d.scale = scale;
    d.edges = edges;
    d.split = split;
    return engine_upload_queries(g->eng, g->stream);
  }
  std::vector<EngQuery> qv(1);
  qv[0] = EngQuery{g->row, edges, split, g->dist, g->n, g->m, 0u, scale, (unsigned)shift, 0u};
  return engine_alloc(g->eng, g->device, g->wt == ADDS_F32, qv, g->grow, g->stream);
}

/* phase engine for plain solves of g (reused while the layout and the kernel
 * variant stay the same) */
static int graph_phase_engine(adds_graph *g, const Knobs &k, int shift, float scale) {
  const uint2 *edges;
  const unsigned *split;
  int rc = graph_layout(g, g->split, k, shift, scale, &edges, &split);
  if (rc) return rc;
  PhQuery q;
  memset(&q, 0, sizeof q);
  q.row = g->row;
  q.edges = edges;
  q.split = split;
  q.dist = g->dist;
  q.n = g->n;
  q.src = 0;
  q.scale = scale;
  q.shift = (unsigned)shift;
  q.m = g->m;
  rc = phase_pull_arrays(g, k, &q);
  if (rc) return rc;
  PhEngine &E = g->peng;
  if (E.nq == 1 && E.variant == (unsigned)k.variant && E.req_group == k.group_ctas &&
      ph_hub_chunk(phase_knobs(k)) >= E.hub_eff) {
    PhQuery &h = E.qs_host[0];
    if (h.edges == edges && h.split == split && h.shift == q.shift && h.scale == scale &&
        h.trow == q.trow)
      return ADDS_OK;
    E.qs_host[0] = q;
    return ph_engine_upload(E, g->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  }
  std::vector<PhQuery> qv(1, q);
  rc = ph_engine_alloc(E, g->device, g->wt == ADDS_F32, qv, phase_knobs(k), g->grow, g->stream);
  if (!rc && g->trace_cap) rc = ph_engine_trace(E, g->trace_cap);
  if (rc) {
    snprintf(g_last_err, sizeof g_last_err, "phase engine allocation failed (%d)", rc);
    ph_engine_free(E);
  }
  return rc;
}

/* Pieces of the rows that one warp of a wave kernel should not relax alone,
 * numbered in whatever order the counter gives.  Depends on the rows only, so
 * it is made once per graph. */
__global__ void k_pieces(const unsigned *row, uint32_t n, unsigned *cnt, unsigned *first,
                         uint4 *piece) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const unsigned r0 = row[v], deg = row[v + 1] - r0;
    if (deg <= WV_PIECE) continue;
    const unsigned k = (deg + WV_PIECE - 1u) / WV_PIECE, c = atomicAdd(cnt, k);
    first[v] = c;
    for (unsigned j = 0; j < k; ++j)
      piece[c + j] = make_uint4(v, r0 + j * WV_PIECE, min(WV_PIECE, deg - j * WV_PIECE), 0u);
  }
}

static int graph_pieces(adds_graph *g) {
  if (g->wpiece || g->max_deg <= WV_PIECE) return ADDS_OK;
  /* a row longer than a piece has fewer than twice as many as its edges fill */
  const size_t cap = 2 * (g->m / WV_PIECE) + 1;
  cudaError_t e = cudaSuccess;
  if (!g->wfirst) e = cudaMalloc(&g->wfirst, ((size_t)g->n + 1) * 4);
  if (e == cudaSuccess) e = cudaMalloc(&g->wpiece, cap * sizeof(uint4));
  unsigned *cnt = g->wfirst ? g->wfirst + g->n : nullptr;
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, 4, g->stream);
  if (e == cudaSuccess) {
    k_pieces<<<592, 256, 0, g->stream>>>(g->row, g->n, cnt, g->wfirst, g->wpiece);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&g->wpieces, cnt, 4, cudaMemcpyDeviceToHost, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) {
    if (g->wpiece) cudaFree(g->wpiece);
    g->wpiece = nullptr;
    return cuda_fail(e, "pieces of long rows");
  }
  g->bytes += ((size_t)g->n + 1) * 4 + cap * sizeof(uint4);
  return ADDS_OK;
}

/* first threshold step of the wave kernels, in distance units */
static float wave_delta(const adds_graph *g, int shift, float scale) {
  const double d = ldexp(1.0, shift);
  return (float)(g->wt == ADDS_F32 ? d / (double)scale : d);
}

/* The edges of a wave kernel's query, and where light ones end.  Light and
 * heavy edges apart: a hub that is improved again within a bucket relaxes its
 * light edges only.  For graphs with long rows that are large enough for edges
 * rather than hops to count (R-MAT 20 0.85 ms against 1.2 with whole rows,
 * R-MAT 18 0.62 both, R-MAT 16 0.49 against 0.41, all on 148 CTAs: the heavy hops
 * are extra, and fewer CTAs make edges count sooner); ER 10^6 x 8 1.0 against
 * 0.56. */
static int wave_layout(adds_graph *g, Split &S, const Knobs &k, int shift, float scale,
                       unsigned ctas, WvQuery *q) {
  q->edges = g->edges;
  q->split = nullptr;
  q->trow = nullptr;
  q->tedges = nullptr;
  if (k.wave != WV_POOL || k.light_heavy == 0 ||
      (k.light_heavy == 2 && (g->max_deg <= WV_PIECE || g->n <= 1771u * ctas)))
    return ADDS_OK;
  int rc = graph_layout(g, S, k, shift, scale, &q->edges, &q->split);
  /* Heavy edges pulled where that reads less, if edges count at all: R-MAT 21 on
   * 148 CTAs 1.11 ms against 1.20, R-MAT 22 1.6 against 1.8, R-MAT 20 0.90 against
   * 0.89; 64 R-MAT 20 queries in groups of 4 18.8 against 21.2. */
  if (!rc && k.pull && (k.pull == 1 || g->m >= 113000ull * ctas)) {
    rc = graph_transposed(g);
    q->trow = g->trow;
    q->tedges = g->tedges;
    q->thr = light_threshold(g, shift, scale);
  }
  return rc;
}

static int graph_wave_engine(adds_graph *g, const Knobs &k, int shift, float scale) {
  const int rp = graph_pieces(g);
  if (rp) return rp;
  WvQuery q;
  memset(&q, 0, sizeof q);
  q.row = g->row;
  const int rl = wave_layout(g, g->split, k, shift, scale,
                             k.group_ctas > 0 ? (unsigned)k.group_ctas : 148u, &q);
  if (rl) return rl;
  q.first = g->wfirst;
  q.piece = g->wpiece;
  q.np = g->wpieces;
  q.dist = g->dist;
  q.n = g->n;
  q.m = g->m;
  q.delta = wave_delta(g, shift, scale);
  WvEngine &E = g->weng;
  const unsigned gs = (unsigned)std::max(0, k.group_ctas);
  if (E.nq == 1 && E.shape == k.wave && E.req_gsize == gs && (E.has_set || !q.split) &&
      (E.kernel == WV_PULL || !q.trow)) {
    const WvQuery &h = E.qs_host[0];
    if (h.delta == q.delta && h.edges == q.edges && h.split == q.split && h.trow == q.trow &&
        h.thr == q.thr) return ADDS_OK;
    E.qs_host[0] = q;
    wv_query_schedule(E.qs_host[0], k.wave);
    return wv_engine_upload(E, g->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  }
  const int rc = wv_engine_alloc(E, g->device, g->wt == ADDS_F32, k.wave, gs,
                                 std::vector<WvQuery>(1, q), g->stream);
  if (rc) snprintf(g_last_err, sizeof g_last_err, "wave kernel allocation failed (%d)", rc);
  return rc;
}

extern "C" int adds_graph_trace(adds_graph *g, uint32_t cap) {
  if (!g || cap > (1u << 24)) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  CK(cudaStreamSynchronize(g->stream));
  g->trace_cap = cap;
  if (g->peng.nq) return ph_engine_trace(g->peng, cap);
  return ADDS_OK;
}

extern "C" int adds_graph_trace_read(adds_graph *g, adds_phase_trace *out, uint32_t cap,
                                     uint64_t *written) {
  if (!g) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  CK(cudaStreamSynchronize(g->stream));
  const uint64_t w = g->peng.nq ? g->peng.g_host->st_trace : 0;
  if (written) *written = w;
  const uint64_t n = std::min<uint64_t>(std::min<uint64_t>(w, g->peng.trace_cap), cap);
  if (out && n) CK(cudaMemcpy(out, g->peng.trace, n * sizeof(PhTrace), cudaMemcpyDeviceToHost));
  return ADDS_OK;
}

static int phase_status(const PhEngine &E) { return ph_engine_status(E, g_last_err, sizeof g_last_err); }

static void fill_phase_stats(const PhEngine &E, adds_stats *s) {
  if (!s) return;
  const PhGlobal &g = *E.g_host;
  s->items_popped = g.st_items;
  s->items_stale = g.st_stale;
  s->edges_scanned = g.st_edges;
  s->pushes = g.st_pushes;
  s->batches = g.st_chunks;
  s->hub_chunks = g.st_hub;
  s->heavy_lists = g.st_heavy;
  for (int i = 0; i < 6; ++i) s->phase_cycles[i] = g.st_cyc[i];
  s->mid_flush_cycles = g.st_cyc[6]; /* grid-phase work */
  s->mid_flushes = g.st_cyc[7];      /* total */
  s->ctas = (int32_t)(E.groups * E.gsize);
  s->engine = ADDS_ENGINE_PHASE;
  /* the launch chain of ph_engine_enqueue when pull phases are possible */
  const bool chain = E.nq == 1 && E.groups == 1 && E.qs_host[0].trow != nullptr;
  s->launches = chain ? (int32_t)(1u + 2u * PH_PULL_SEGMENTS) : 1;
  s->phases = g.st_phases;
  s->solo_phases = g.st_solo;
  s->repushes = g.st_repush;
}

static void fill_wave_stats(const WvEngine &E, adds_stats *s) {
  if (!s) return;
  const WvStat &t = *E.st_host;
  s->items_popped = t.items;
  s->items_stale = t.stale;
  s->edges_scanned = t.edges;
  s->pushes = t.pushes;
  s->phases = t.steps;
  s->batches = t.splits;
  s->ctas = (int32_t)E.ctas;
  s->launches = E.fills ? 2 : 1;
}

/* error word, reset and counters of whatever ran g's last solves */
static int graph_status(const adds_graph *g) {
  if (g->last_wave) return wv_engine_status(g->weng, g_last_err, sizeof g_last_err);
  return g->last_engine == ADDS_ENGINE_PHASE ? phase_status(g->peng) : engine_status(g->eng);
}
static void graph_reset(adds_graph *g, cudaStream_t st) {
  if (g->last_wave) wv_engine_reset(g->weng, st);
  else if (g->last_engine == ADDS_ENGINE_PHASE) ph_engine_reset(g->peng, st);
  else engine_full_reset(g->eng, st);
}
/* after a worklist overflow: a larger pool on the rerun, or, for the wave
 * kernels, whose lists are sized once, the engine that has one */
static void graph_outgrown(adds_graph *g) {
  if (g->last_wave) {
    g->wave_off = true;
    wv_engine_free(g->weng);
    return;
  }
  g->grow *= 2;
  if (g->last_engine == ADDS_ENGINE_PHASE) ph_engine_free(g->peng); else engine_free(g->eng);
}
static void graph_stats(const adds_graph *g, adds_stats *stats, double ms, double kms) {
  if (!stats) return;
  memset(stats, 0, sizeof *stats);
  stats->ms = ms;
  stats->kernel_ms = kms;
  if (g->last_wave) {
    fill_wave_stats(g->weng, stats);
    stats->engine = g->last_engine;
    stats->delta_shift = g->last_shift;
  } else if (g->last_engine == ADDS_ENGINE_PHASE) {
    fill_phase_stats(g->peng, stats);
    stats->delta_shift = (int32_t)g->peng.qs_host[0].shift;
  } else {
    fill_stats(g->eng, g->last_params, stats);
    stats->delta_shift = (int32_t)g->eng.qs_host[0].shift0;
    stats->engine = ADDS_ENGINE_ASYNC;
  }
}

static cudaStream_t pick_stream(const adds_graph *g, const adds_opts *o) {
  return (o && o->stream) ? (cudaStream_t)o->stream : g->stream;
}

/* The wave kernel of a plain solve whose schedule is left to the library, or
 * none.  Measured on one B200, untuned solves with automatic knobs (wave
 * kernel against the phase engine, which they ran on before; the asynchronous
 * engine in brackets):
 *   average degree under 6: 64^2 grid 0.25 against 2.2 ms (0.58), 300^2 0.88
 *   against 14.9 (1.8), 4096^2 18.3 against 310 (38); one CTA below 4,096
 *   vertices, where a group's exchanges cost what its width saves (16^2 0.107
 *   against 0.118, 64^2 0.295 against 0.25);
 *   longer rows: ER 4,001 x 8 0.16 against 0.57 (0.29), ER 10^6 x 8 0.56 against
 *   1.7 (0.95), ER 8 x 10^6 x 16 2.3 against 4.4, R-MAT 16 0.40 against 0.84
 *   (0.49), R-MAT 20 0.89 against 1.8 (1.15), R-MAT 22 1.6 against 2.0, float 1.9
 *   against 2.4, R-MAT 23 2.3 against 2.4 with weights up to 1,000, 1.7 against 2.2
 *   up to 10; R-MAT 24 4.5 against 4.2 up to 10,000, 3.6 both up to 1,000: from
 *   2^27 edges on, graphs with long rows stay with the phase engine. */
static int auto_wave(const adds_graph *g, const adds_opts *o) {
  if (g->wave_off || g->trace_cap || g->tuned || !schedule_auto(o)) return -1;
  if (g->avg_deg < 6.0 && g->m < (1ull << 31)) return g->n < 4096u ? WV_WIDE : WV_GROUP;
  if (g->n < 32768u && g->max_deg <= WV_PIECE) return WV_GROUP; /* ER 4,001 x 8: 0.15, pooled 0.18 */
  return g->m < (g->max_deg <= WV_PIECE ? 1ull << 29 : 1ull << 27) ? WV_POOL : -1;
}

/* The bucket of a pooled wave kernel that relaxes light and heavy edges apart,
 * no narrower than auto_shift's.  Where rows are long, the 4 avg_w / degree of
 * auto_shift is too narrow above a degree of 8: the heavy edges that a wide
 * bucket saves for later are most of the rows at any of these degrees.  Best
 * over degrees 8 to 64, scales 17 to 22 and seven weight ranges: 0.44 of a
 * mean weight, a quarter once the heavy edges are pulled, less from some 90
 * million edges on (R-MAT 18 x 16 0.68 -> 0.58 ms, 18 x 64 1.35 -> 0.98, 20 x 16 0.99
 * -> 0.94, 20 x 32 1.55 -> 1.10, 21 x 32 1.73 -> 1.48 with weights up to 10,000; up
 * to 10 and 100 it saves more, for floats less: 19 x 32 with a = 0.7 loses 6 %,
 * 22 x 24 lost 13 % at a quarter).  Integer weights have one added, so that
 * few-valued ones have light edges.  Not below 664
 * vertices a CTA, where the rows are relaxed whole and there is little to
 * settle (R-MAT 16 0.34 -> 0.36; R-MAT 17 0.50 -> 0.48), nor without long rows (ER
 * 10^6 x 32 0.73 at auto_shift's 2^9, 1.3 at 2^11). */
static int pooled_shift(const adds_graph *g, int shift) {
  constexpr unsigned ctas = 148;
  if (g->max_deg <= WV_PIECE || g->n <= 664u * ctas) return shift;
  const double c = g->m >= 610000ull * ctas ? 0.175 : g->m >= 113000ull * ctas ? 0.25 : 0.44;
  const double keys = g->wt == ADDS_F32 ? c * 65536.0 : c * g->avg_w + 1.0;
  return std::max(shift, std::min(31, (int)lround(log2(keys))));
}

/* Enqueues one solve; no host synchronisation.  Each solve records four
 * events (start, solver start, solver end, end) in the graph's ring. */
static int sssp_enqueue(adds_graph *g, uint32_t src, const adds_opts *opts) {
  int shift;
  float scale;
  Knobs k;
  adds_opts tw;
  const adds_opts *o = opts;
  if (g->tuned && g->tuned_wave.wave > 0 && !g->wave_off && !g->trace_cap && schedule_auto(opts)) {
    tw = g->tuned_wave;
    if (opts) tw.timeout_ms = opts->timeout_ms;
    o = &tw;
  }
  resolve(g, o, &k, &shift, &scale);
  if (k.wave < 0) {
    k.wave = auto_wave(g, opts);
    if (k.wave == WV_POOL) shift = pooled_shift(g, shift);
  }
  if (g->wave_off) k.wave = -1;
  const bool phase = k.engine == ADDS_ENGINE_PHASE, wave = k.wave >= 0;
  int rc = ADDS_OK;
  if (wave) {
    rc = graph_wave_engine(g, k, shift, scale);
    if (rc == ADDS_ERR_OOM || rc == ADDS_ERR_UNSUPPORTED) { /* no room for its lists */
      g->wave_off = true;
      return sssp_enqueue(g, src, opts);
    }
  } else {
    rc = phase ? graph_phase_engine(g, k, shift, scale) : graph_engine(g, k, shift, scale);
  }
  if (rc) return rc;
  cudaStream_t st = pick_stream(g, opts);
  g->last_knobs = k;
  g->last_engine = k.engine;
  g->last_wave = wave;
  g->last_shift = shift;
  if (g->ring_used == adds_graph::kRing) { /* ring full: fold into nothing */
    CK(cudaStreamSynchronize(st));
    g->ring_used = 0;
  }
  cudaEvent_t *ev = g->ring[g->ring_used];
  for (int j = 0; j < 4; ++j)
    if (!ev[j]) CK(cudaEventCreate(&ev[j]));
  CK(cudaEventRecord(ev[0], st));
  if (wave) {
    if (wv_engine_enqueue(g->weng, src, k.timeout_ns, st, ev[1], ev[2]))
      return cuda_fail(cudaGetLastError(), "wave kernel launch");
  } else if (phase) {
    PhParams P;
    if (ph_engine_params(g->peng, phase_knobs(k), src, &P)) return ADDS_ERR_INVALID;
    g->last_pp = P;
    rc = ph_engine_enqueue(g->peng, P, st, ev[1], ev[2]);
    if (rc) return cuda_fail(cudaGetLastError(), "phase engine launch");
  } else {
    EngParams P = make_params(g->eng, k, src);
    g->last_params = P;
    rc = engine_enqueue(g->eng, P, st, ev[1], ev[2]);
  }
  if (rc) return rc;
  CK(cudaEventRecord(ev[3], st));
  ++g->ring_used;
  return ADDS_OK;
}

/* total and solver-kernel time of the solves in the ring (stream synced) */
static void ring_times(adds_graph *g, double *ms, double *kms) {
  double a = 0, b = 0;
  for (int i = 0; i < g->ring_used; ++i) {
    float x = 0, y = 0;
    cudaEventElapsedTime(&x, g->ring[i][0], g->ring[i][3]);
    cudaEventElapsedTime(&y, g->ring[i][1], g->ring[i][2]);
    a += x;
    b += y;
  }
  cudaGetLastError();
  g->ring_used = 0;
  *ms = a;
  *kms = b;
}

extern "C" int adds_sssp(adds_graph *g, uint32_t src, void *dist_out, const adds_opts *opts,
                         adds_stats *stats) {
  if (!g || src >= g->n) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  cudaStream_t st = pick_stream(g, opts);
  int retries = 0;
  CK(cudaStreamSynchronize(st));
  g->ring_used = 0;
  g->pend.clear();
  for (;;) {
    rc = sssp_enqueue(g, src, opts);
    if (rc) return rc;
    CK(cudaStreamSynchronize(st));
    rc = graph_status(g);
    if (rc == ADDS_ERR_WL_OVERFLOW && retries < 4) {
      ++retries;
      graph_outgrown(g); /* re-allocated at the larger size on the rerun */
      g->ring_used = 0;
      continue;
    }
    if (rc) {
      graph_reset(g, st);
      g->ring_used = 0;
      return rc;
    }
    break;
  }
  double ms = 0, kms = 0;
  ring_times(g, &ms, &kms);
  graph_stats(g, stats, ms, kms);
  if (stats) stats->retries = retries;
  g->pending = 0;
  if (dist_out) return adds_graph_last_dist(g, dist_out);
  return ADDS_OK;
}

/* Solves srcs[0..ns) one after another and copies result i to dist_out[i]
 * while solve i+1 runs: the result is copied on the device into one of two
 * staging buffers, and a second stream moves it to host memory, so the
 * device-to-host transfer overlaps the next solve instead of following it.
 * The host loop enqueues solve i before it hands result i-1 to the copy
 * stream, so a pageable destination (whose copy blocks the host) overlaps
 * as well.  A device destination is copied on the solve stream. */
extern "C" int adds_sssp_sources(adds_graph *g, const uint32_t *srcs, uint32_t ns,
                                 void *const *dist_out, const adds_opts *opts,
                                 adds_stats *stats) {
  if (!g || (ns && (!srcs || !dist_out))) return ADDS_ERR_INVALID;
  for (uint32_t i = 0; i < ns; ++i)
    if (srcs[i] >= g->n || !dist_out[i]) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  if (ns == 0) return ADDS_OK;
  const size_t bytes = (size_t)g->n * 4;
  cudaStream_t st = pick_stream(g, opts);
  CK(cudaStreamSynchronize(st));
  g->ring_used = 0;
  g->pend.clear();
  if (!g->stage) {
    CK(cudaMalloc(&g->stage, 2 * (bytes ? bytes : 4)));
    g->bytes += 2 * bytes;
  }
  if (!g->cstream) CK(cudaStreamCreateWithFlags(&g->cstream, cudaStreamNonBlocking));
  for (int j = 0; j < 2; ++j) {
    if (!g->ev_free[j]) CK(cudaEventCreateWithFlags(&g->ev_free[j], cudaEventDisableTiming));
    if (!g->ev_ready[j]) CK(cudaEventCreateWithFlags(&g->ev_ready[j], cudaEventDisableTiming));
  }
  bool staged[2] = {false, false};
  /* result i, staged in buffer i & 1, to the caller on the copy stream */
  auto copy_out = [&](uint32_t i) -> int {
    const int j = (int)(i & 1u);
    CK(cudaStreamWaitEvent(g->cstream, g->ev_ready[j], 0));
    CK(cudaMemcpyAsync(dist_out[i], g->stage + (size_t)j * g->n, bytes,
                       cudaMemcpyDeviceToHost, g->cstream));
    CK(cudaEventRecord(g->ev_free[j], g->cstream));
    return ADDS_OK;
  };
  int pending_out = -1; /* the staged result not yet handed to the copy stream */
  for (uint32_t i = 0; i < ns && !rc; ++i) {
    rc = sssp_enqueue(g, srcs[i], opts);
    if (rc) break;
    /* solve i is queued: now the previous result may leave */
    if (pending_out >= 0) {
      rc = copy_out((uint32_t)pending_out);
      pending_out = -1;
      if (rc) break;
    }
    if (is_device_ptr(dist_out[i])) {
      CK(cudaMemcpyAsync(dist_out[i], g->dist, bytes, cudaMemcpyDeviceToDevice, st));
      continue;
    }
    const int j = (int)(i & 1u);
    if (staged[j]) CK(cudaStreamWaitEvent(st, g->ev_free[j], 0));
    CK(cudaMemcpyAsync(g->stage + (size_t)j * g->n, g->dist, bytes, cudaMemcpyDeviceToDevice,
                       st));
    CK(cudaEventRecord(g->ev_ready[j], st));
    staged[j] = true;
    pending_out = (int)i;
  }
  if (!rc && pending_out >= 0) rc = copy_out((uint32_t)pending_out);
  const cudaError_t e1 = cudaStreamSynchronize(st);
  const cudaError_t e2 = cudaStreamSynchronize(g->cstream);
  if (rc) {
    g->ring_used = 0;
    return rc;
  }
  if (e1 != cudaSuccess || e2 != cudaSuccess)
    return cuda_fail(e1 != cudaSuccess ? e1 : e2, "multi-source solve");
  rc = graph_status(g);
  if (rc == ADDS_ERR_WL_OVERFLOW) {
    /* the worklist outgrew its pool: solve one at a time, which regrows it */
    g->ring_used = 0;
    graph_reset(g, st);
    for (uint32_t i = 0; i < ns; ++i) {
      rc = adds_sssp(g, srcs[i], dist_out[i], opts, i + 1 == ns ? stats : nullptr);
      if (rc) return rc;
    }
    return ADDS_OK;
  }
  if (rc) {
    graph_reset(g, st);
    g->ring_used = 0;
    return rc;
  }
  double ms = 0, kms = 0;
  ring_times(g, &ms, &kms);
  graph_stats(g, stats, ms, kms);
  g->pending = 0;
  return ADDS_OK;
}

/* Asynchronous form for back-to-back solves: errors surface in
 * adds_graph_sync (a failed solve makes the following ones exit at once). */
extern "C" int adds_sssp_async(adds_graph *g, uint32_t src, const adds_opts *opts) {
  if (!g || src >= g->n) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  rc = sssp_enqueue(g, src, opts);
  if (!rc) {
    ++g->pending;
    adds_opts o;
    if (opts) o = *opts; else adds_opts_init(&o);
    g->pend.emplace_back(src, o);
  }
  return rc;
}

extern "C" int adds_graph_sync(adds_graph *g, adds_stats *stats) {
  if (!g) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  CK(cudaStreamSynchronize(g->stream));
  double ms = 0, kms = 0;
  ring_times(g, &ms, &kms);
  const bool phase = g->last_engine == ADDS_ENGINE_PHASE;
  if (g->last_wave ? g->weng.nq == 0 : phase ? g->peng.nq == 0 : g->eng.nq == 0) return ADDS_OK;
  rc = graph_status(g);
  g->pending = 0;
  std::vector<std::pair<uint32_t, adds_opts>> redo;
  redo.swap(g->pend);
  if (rc == ADDS_ERR_WL_OVERFLOW && !redo.empty()) {
    /* a solve outgrew the worklist pool (and the ones after it exited):
     * run them all again one at a time, as adds_sssp does, on a larger pool;
     * the graph then holds the last one's distances as it would have */
    graph_outgrown(g);
    for (size_t i = 0; i < redo.size(); ++i) {
      rc = adds_sssp(g, redo[i].first, nullptr, &redo[i].second,
                     i + 1 == redo.size() ? stats : nullptr);
      if (rc) return rc;
    }
    return ADDS_OK;
  }
  if (rc) {
    graph_reset(g, g->stream);
    return rc;
  }
  graph_stats(g, stats, ms, kms);
  return ADDS_OK;
}

extern "C" int adds_graph_last_dist(adds_graph *g, void *dist_out) {
  if (!g || !dist_out) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(g->device));
  const bool dev = is_device_ptr(dist_out);
  CK(cudaMemcpyAsync(dist_out, g->dist, (size_t)g->n * 4,
                     dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, g->stream));
  CK(cudaStreamSynchronize(g->stream));
  return ADDS_OK;
}

extern "C" int adds_graph_reached(adds_graph *g, uint64_t *reached, uint64_t *reached_edges) {
  if (!g) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(g->device));
  unsigned long long *d = nullptr, h[2] = {0, 0};
  CK(cudaMalloc(&d, 16));
  CK(cudaMemsetAsync(d, 0, 16, g->stream));
  CK(adds_engine_launch_reached(g->row, g->dist, g->n,
                                g->wt == ADDS_F32 ? ADDS_INF_F32_BITSV : ADDS_INF_I32_BITS, d,
                                g->stream));
  CK(cudaMemcpyAsync(h, d, 16, cudaMemcpyDeviceToHost, g->stream));
  CK(cudaStreamSynchronize(g->stream));
  cudaFree(d);
  if (reached) *reached = h[0];
  if (reached_edges) *reached_edges = h[1];
  return ADDS_OK;
}

/* ------------------------------------------------------------------------ */
/* batches                                                                    */
struct adds_batch {
  int device = 0;
  bool flt = false;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::vector<adds_graph *> qgraph;
  std::vector<uint32_t> srcs;
  std::vector<adds_graph *> ugraph; /* distinct graphs, first-use order */
  std::vector<unsigned> qgid;
  std::vector<Split> splits; /* one per distinct graph, whose queries share a width */
  unsigned *dist_all = nullptr;
  std::vector<size_t> dist_off;
  Engine eng;
  PhEngine peng; /* used when kn.engine is ADDS_ENGINE_PHASE */
  WvEngine weng; /* used when kn.wave names a variant */
  unsigned wave_group = 0; /* CTAs per query of its group variants */
  PhParams pp;
  unsigned grow = 1;
  Knobs kn;
  std::vector<int> shifts;
  std::vector<float> scales;
  cudaGraphExec_t exec = nullptr;
  bool captured = false;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, k0 = nullptr, k1 = nullptr;
  EngParams P;
  void *adj = nullptr; /* backward scratch (adjoint.cu) */
  std::vector<unsigned long long> wversions; /* graph weight versions seen */
};

static int batch_phase_engine(adds_batch *b) {
  std::vector<PhQuery> qv(b->qgraph.size());
  for (size_t i = 0; i < qv.size(); ++i) {
    adds_graph *g = b->qgraph[i];
    const uint2 *edges;
    const unsigned *split;
    const int rc = graph_layout(g, b->splits[b->qgid[i]], b->kn, b->shifts[i], b->scales[i], &edges,
                                &split);
    if (rc) return rc;
    PhQuery q;
    memset(&q, 0, sizeof q);
    q.row = g->row;
    q.edges = edges;
    q.split = split;
    q.dist = b->dist_all + b->dist_off[i];
    q.n = g->n;
    q.src = b->srcs[i];
    q.scale = b->scales[i];
    q.shift = (unsigned)b->shifts[i];
    q.m = g->m;
    /* a pull phase ends a launch, which the groups of a batch do not share:
     * only a batch of one query pulls */
    if (qv.size() == 1) {
      const int rp = phase_pull_arrays(g, b->kn, &q);
      if (rp) return rp;
    }
    qv[i] = q;
  }
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  b->captured = false;
  const PhKnobs pk = phase_knobs(b->kn);
  int rc = ph_engine_alloc(b->peng, b->device, b->flt, qv, pk, b->grow, b->stream);
  if (rc) {
    snprintf(g_last_err, sizeof g_last_err, "phase engine allocation failed (%d)", rc);
    ph_engine_free(b->peng);
    return rc;
  }
  ph_engine_params(b->peng, pk, 0xFFFFFFFFu, &b->pp);
  return ADDS_OK;
}

static int batch_wave_engine(adds_batch *b) {
  std::vector<WvQuery> qv(b->qgraph.size());
  for (size_t i = 0; i < qv.size(); ++i) {
    adds_graph *g = b->qgraph[i];
    const int rp = graph_pieces(g);
    if (rp) return rp;
    WvQuery q;
    memset(&q, 0, sizeof q);
    q.row = g->row;
    const int rl = wave_layout(g, b->splits[b->qgid[i]], b->kn, b->shifts[i], b->scales[i],
                               b->wave_group, &q);
    if (rl) return rl;
    q.first = g->wfirst;
    q.piece = g->wpiece;
    q.np = g->wpieces;
    q.dist = b->dist_all + b->dist_off[i];
    q.n = g->n;
    q.m = g->m;
    q.src = b->srcs[i];
    q.delta = wave_delta(g, b->shifts[i], b->scales[i]);
    qv[i] = q;
  }
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  b->captured = false;
  const int rc = wv_engine_alloc(b->weng, b->device, b->flt, b->kn.wave, b->wave_group, qv, b->stream);
  if (rc) snprintf(g_last_err, sizeof g_last_err, "wave kernel allocation failed (%d)", rc);
  return rc;
}

static int batch_engine(adds_batch *b) {
  b->wversions.clear();
  for (adds_graph *g : b->ugraph) b->wversions.push_back(g->wversion);
  if (b->kn.wave >= 0) {
    const int rw = batch_wave_engine(b);
    if (rw != ADDS_ERR_OOM && rw != ADDS_ERR_UNSUPPORTED) return rw;
    b->kn.wave = -1; /* no room for its lists */
  }
  if (b->kn.engine == ADDS_ENGINE_PHASE) return batch_phase_engine(b);
  std::vector<EngQuery> qv(b->qgraph.size());
  for (size_t i = 0; i < qv.size(); ++i) {
    adds_graph *g = b->qgraph[i];
    const uint2 *edges;
    const unsigned *split;
    const int rc = graph_layout(g, b->splits[b->qgid[i]], b->kn, b->shifts[i], b->scales[i], &edges,
                                &split);
    if (rc) return rc;
    qv[i] = EngQuery{g->row, edges, split, b->dist_all + b->dist_off[i], g->n, g->m, b->srcs[i],
                     b->scales[i], (unsigned)b->shifts[i], b->qgid[i]};
  }
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  b->captured = false;
  int rc = engine_alloc(b->eng, b->device, b->flt, qv, b->grow, b->stream);
  if (rc) {
    engine_free(b->eng);
    return rc;
  }
  b->P = make_params(b->eng, b->kn, 0xFFFFFFFFu);
  return ADDS_OK;
}

extern "C" void adds_batch_free(adds_batch *b);
void adds_adjoint_free(void *adj);

extern "C" int adds_batch_create(adds_graph *const *graphs, const uint32_t *srcs, uint32_t nq,
                                 const adds_opts *opts, adds_batch **out) {
  if (!graphs || !srcs || !out || nq == 0 || nq > 65535) return ADDS_ERR_INVALID;
  *out = nullptr;
  const int dev = graphs[0]->device;
  const adds_wtype wt = graphs[0]->wt;
  for (uint32_t i = 0; i < nq; ++i) {
    if (!graphs[i] || graphs[i]->device != dev || graphs[i]->wt != wt || srcs[i] >= graphs[i]->n)
      return ADDS_ERR_INVALID;
  }
  int rc = set_device(dev);
  if (rc) return rc;
  adds_batch *b = new adds_batch();
  b->device = dev;
  b->flt = wt == ADDS_F32;
  if (opts && opts->stream) b->stream = (cudaStream_t)opts->stream;
  else {
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      delete b;
      return ADDS_ERR_CUDA;
    }
    b->own_stream = true;
  }
  b->qgraph.assign(graphs, graphs + nq);
  b->srcs.assign(srcs, srcs + nq);
  size_t tot = 0;
  b->dist_off.resize(nq);
  b->shifts.resize(nq);
  b->scales.resize(nq);
  /* Bucket widths are per query (a graph's tuned width, else the
   * heuristic).  The launch-wide knobs (engine, kernel variant, window, CTA
   * counts...) are the caller's, else the defaults: a graph's tuned knobs
   * are for a plain solve that has the whole GPU, while a batch runs many
   * queries side by side.  The engine, unless the caller names one, follows
   * the largest query's graph: the asynchronous engine for a sparse,
   * high-diameter graph (average degree under 6: grids, road networks),
   * the phase engine otherwise.  Measured on the batched configurations:
   * 256 R-MAT 20 and ER queries 7,719 solves/s on the phase engine against
   * 4,669 on the asynchronous one (which a plain solve on R-MAT 20 may
   * tune to); 2,048 queries on 128 grids 124-163 ms forward on the
   * asynchronous engine against 626 ms on the phase engine. */
  uint32_t big = 0;
  for (uint32_t i = 1; i < nq; ++i)
    if ((uint64_t)graphs[i]->n + graphs[i]->m > (uint64_t)graphs[big]->n + graphs[big]->m) big = i;
  for (uint32_t i = 0; i < nq; ++i) {
    adds_graph *g = graphs[i];
    auto it = std::find(b->ugraph.begin(), b->ugraph.end(), g);
    unsigned gid = (unsigned)(it - b->ugraph.begin());
    if (it == b->ugraph.end()) b->ugraph.push_back(g);
    b->qgid.push_back(gid);
    b->dist_off[i] = tot;
    tot += ((size_t)g->n + 31) & ~(size_t)31;
    Knobs k;
    resolve(g, opts, &k, &b->shifts[i], &b->scales[i]);
  }
  b->splits.resize(b->ugraph.size());
  {
    adds_opts lw;
    if (opts) lw = *opts; else adds_opts_init(&lw);
    if (lw.engine <= 0)
      lw.engine = graphs[big]->avg_deg < 6.0 ? ADDS_ENGINE_ASYNC : ADDS_ENGINE_PHASE;
    int s_unused;
    float sc_unused;
    resolve(graphs[big], &lw, &b->kn, &s_unused, &sc_unused, false);
    /* With the schedule left to the library, the wave kernels (against the
     * engine they stand in for).  Sparse graphs: four SMs or more a query while
     * there are enough (15 queries on grids of side 61 to 130 0.47 ms, one SM
     * each 0.53), an SM each up to 148 queries (60 on a 257 x 255 road 1.6 ms, two
     * SMs each 2.0, the asynchronous engine 4.7), else four queries to an SM (128
     * grids x 16 sources 7.3 ms against 98).  Others: groups of at least four SMs,
     * which take the queries one after another (192 ER graphs and 64 sources on
     * R-MAT 20 in groups of 1, 2, 4, 6, 9, 18: 38, 23.5, 21.9, 22.3, 22.8, 26.4 ms
     * before pulls, 18.8 in groups of 4 with them; phase engine 27.6). */
    if (b->kn.wave < 0 && schedule_auto(opts)) {
      bool sparse = true, fits = true;
      for (adds_graph *g : b->ugraph) {
        sparse = sparse && g->avg_deg < 6.0;
        fits = fits && g->m < (1ull << 27);
      }
      if (sparse) b->kn.wave = nq <= 37u ? WV_GROUP : (nq <= 148u ? WV_WIDE : WV_CTA);
      else if (fits) b->kn.wave = WV_POOL;
    }
    if (b->kn.wave >= WV_GROUP) {
      int sms = 0;
      CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      b->wave_group = opts && opts->group_ctas > 0 ? (unsigned)opts->group_ctas
                                                    : std::max(4u, (unsigned)sms / nq);
    }
  }
  /* the batch sizes its groups itself unless the caller says otherwise */
  b->kn.group_ctas = (opts && opts->group_ctas > 0) ? opts->group_ctas : 0;
  if (cudaMalloc(&b->dist_all, tot * 4) != cudaSuccess ||
      cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess ||
      cudaEventCreate(&b->k0) != cudaSuccess || cudaEventCreate(&b->k1) != cudaSuccess) {
    cudaGetLastError();
    adds_batch_free(b);
    return ADDS_ERR_OOM;
  }
  rc = batch_engine(b);
  if (rc) {
    adds_batch_free(b);
    return rc;
  }
  *out = b;
  return ADDS_OK;
}

extern "C" void adds_batch_free(adds_batch *b) {
  if (!b) return;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  engine_free(b->eng);
  ph_engine_free(b->peng);
  wv_engine_free(b->weng);
  for (Split &s : b->splits)
    if (s.at) cudaFree(s.at);
  if (b->dist_all) cudaFree(b->dist_all);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->k0) cudaEventDestroy(b->k0);
  if (b->k1) cudaEventDestroy(b->k1);
  if (b->adj) adds_adjoint_free(b->adj);
  if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

/* false between a failed layout (no memory, say) and the next launch */
static bool batch_ready(const adds_batch *b) {
  return (b->kn.wave >= 0 ? b->weng.nq : b->kn.engine == ADDS_ENGINE_PHASE ? b->peng.nq : b->eng.nq) != 0;
}
static int batch_status(const adds_batch *b) {
  if (b->kn.wave >= 0) return wv_engine_status(b->weng, g_last_err, sizeof g_last_err);
  return b->kn.engine == ADDS_ENGINE_PHASE ? phase_status(b->peng) : engine_status(b->eng);
}
static void batch_reset(adds_batch *b) {
  if (b->kn.wave >= 0) wv_engine_reset(b->weng, b->stream);
  else if (b->kn.engine == ADDS_ENGINE_PHASE) ph_engine_reset(b->peng, b->stream);
  else engine_full_reset(b->eng, b->stream);
}

/* init + solve + status read-back, captured once as a CUDA graph */
static int batch_capture(adds_batch *b) {
  cudaGraph_t gr = nullptr;
  CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  int rc = b->kn.wave >= 0
               ? (wv_engine_enqueue(b->weng, 0xFFFFFFFFu, b->kn.timeout_ns, b->stream, b->k0, b->k1)
                      ? ADDS_ERR_CUDA
                      : ADDS_OK)
           : b->kn.engine == ADDS_ENGINE_PHASE
               ? (ph_engine_enqueue(b->peng, b->pp, b->stream, b->k0, b->k1) ? ADDS_ERR_CUDA : ADDS_OK)
               : engine_enqueue(b->eng, b->P, b->stream, b->k0, b->k1);
  cudaError_t e = cudaStreamEndCapture(b->stream, &gr);
  if (rc || e != cudaSuccess) {
    if (gr) cudaGraphDestroy(gr);
    cudaGetLastError();
    return rc ? rc : cuda_fail(e, "capture");
  }
  e = cudaGraphInstantiate(&b->exec, gr, 0);
  cudaGraphDestroy(gr);
  if (e != cudaSuccess) return cuda_fail(e, "instantiate");
  b->captured = true;
  return ADDS_OK;
}

/* weights changed since the descriptors were built: the weight-sorted
 * copies are rebuilt and the descriptors re-pointed (same sizing) */
static int batch_relayout(adds_batch *b) {
  bool changed = false;
  for (size_t i = 0; i < b->ugraph.size(); ++i)
    if (b->ugraph[i]->wversion != b->wversions[i]) changed = true;
  if (!changed) return ADDS_OK;
  if (b->kn.wave >= 0) { /* the CSR itself, or the copy sorted by weight */
    bool moved = false;
    for (size_t i = 0; i < b->qgraph.size(); ++i) {
      WvQuery &q = b->weng.qs_host[i];
      const WvQuery was = q;
      const int rc = wave_layout(b->qgraph[i], b->splits[b->qgid[i]], b->kn, b->shifts[i],
                                 b->scales[i], b->wave_group, &q);
      if (rc) return rc;
      moved = moved || q.edges != was.edges || q.split != was.split || q.trow != was.trow ||
              q.thr != was.thr;
    }
    for (size_t i = 0; i < b->ugraph.size(); ++i) b->wversions[i] = b->ugraph[i]->wversion;
    return moved && wv_engine_upload(b->weng, b->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  }
  for (size_t i = 0; i < b->qgraph.size(); ++i) {
    const uint2 *edges;
    const unsigned *split;
    const int rc = graph_layout(b->qgraph[i], b->splits[b->qgid[i]], b->kn, b->shifts[i],
                                b->scales[i], &edges, &split);
    if (rc) return rc;
    if (b->kn.engine == ADDS_ENGINE_PHASE) {
      PhQuery &q = b->peng.qs_host[i];
      q.edges = edges;
      q.split = split;
      if (b->qgraph.size() == 1) { /* new weights for the in-edge copy */
        const int rp = phase_pull_arrays(b->qgraph[i], b->kn, &q);
        if (rp) return rp;
      }
    } else {
      b->eng.qs_host[i].edges = edges;
      b->eng.qs_host[i].split = split;
    }
  }
  for (size_t i = 0; i < b->ugraph.size(); ++i) b->wversions[i] = b->ugraph[i]->wversion;
  if (b->kn.engine == ADDS_ENGINE_PHASE)
    return ph_engine_upload(b->peng, b->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  return engine_upload_queries(b->eng, b->stream);
}

extern "C" int adds_batch_launch(adds_batch *b) {
  if (!b) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(b->device));
  const int rl = batch_ready(b) ? batch_relayout(b) : batch_engine(b);
  if (rl) return rl;
  if (!b->captured) {
    int rc = batch_capture(b);
    if (rc) return rc;
  }
  CK(cudaEventRecord(b->ev0, b->stream));
  CK(cudaGraphLaunch(b->exec, b->stream));
  CK(cudaEventRecord(b->ev1, b->stream));
  return ADDS_OK;
}

/* Waits for the launches in flight.  The wave kernels' lists do not grow: after
 * an overflow the batch is laid out for its engine, from then on, and what was
 * launched is solved there (*moved is set). */
static int batch_wait(adds_batch *b, bool *moved) {
  *moved = false;
  CK(cudaStreamSynchronize(b->stream));
  if (!batch_ready(b)) return ADDS_ERR_INVALID;
  int rc = batch_status(b);
  if (rc != ADDS_ERR_WL_OVERFLOW || b->kn.wave < 0) return rc;
  *moved = true;
  wv_engine_free(b->weng);
  b->kn.wave = -1;
  rc = adds_batch_launch(b);
  if (rc) return rc;
  CK(cudaStreamSynchronize(b->stream));
  return batch_status(b);
}

extern "C" int adds_batch_sync(adds_batch *b, adds_stats *stats) {
  if (!b) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(b->device));
  bool moved;
  const int rc = batch_wait(b, &moved);
  const bool phase = b->kn.engine == ADDS_ENGINE_PHASE;
  if (rc) {
    if (batch_ready(b)) batch_reset(b); /* reported: the next launch starts from a clean engine */
    return rc;
  }
  if (stats) {
    memset(stats, 0, sizeof *stats);
    float ms = 0, kms = 0;
    CK(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
    CK(cudaEventElapsedTime(&kms, b->k0, b->k1));
    stats->ms = ms;
    stats->kernel_ms = kms;
    if (b->kn.wave >= 0) {
      fill_wave_stats(b->weng, stats);
      stats->engine = b->kn.engine;
    } else if (phase) {
      fill_phase_stats(b->peng, stats);
    } else {
      fill_stats(b->eng, b->P, stats);
      stats->engine = ADDS_ENGINE_ASYNC;
    }
    stats->delta_shift = b->shifts.empty() ? 0 : b->shifts[0];
    stats->retries = moved ? 1 : 0;
  }
  return ADDS_OK;
}

extern "C" int adds_batch_run(adds_batch *b, adds_stats *stats) {
  if (!b) return ADDS_ERR_INVALID;
  int retries = 0;
  for (;;) {
    int rc = adds_batch_launch(b);
    if (rc) return rc;
    rc = adds_batch_sync(b, stats);
    if (rc == ADDS_ERR_WL_OVERFLOW && retries < 4) {
      ++retries;
      b->grow *= 2;
      rc = batch_engine(b);
      if (rc) return rc;
      continue;
    }
    if (rc) return rc;
    if (stats) stats->retries += retries;
    return ADDS_OK;
  }
}

extern "C" int adds_batch_set_sources(adds_batch *b, const uint32_t *srcs) {
  if (!b || !srcs) return ADDS_ERR_INVALID;
  for (size_t i = 0; i < b->srcs.size(); ++i)
    if (srcs[i] >= b->qgraph[i]->n) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(b->device));
  /* a launch that overflowed is solved with the sources it had */
  bool moved;
  const int rw = batch_wait(b, &moved);
  if (moved && rw) return rw;
  for (size_t i = 0; i < b->srcs.size(); ++i) b->srcs[i] = srcs[i];
  if (!batch_ready(b)) return ADDS_OK; /* the next launch lays them out */
  if (b->kn.wave >= 0) {
    for (size_t i = 0; i < b->srcs.size(); ++i) b->weng.qs_host[i].src = srcs[i];
    return wv_engine_upload(b->weng, b->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  }
  if (b->kn.engine == ADDS_ENGINE_PHASE) {
    for (size_t i = 0; i < b->srcs.size(); ++i) b->peng.qs_host[i].src = srcs[i];
    return ph_engine_upload(b->peng, b->stream) ? ADDS_ERR_CUDA : ADDS_OK;
  }
  for (size_t i = 0; i < b->srcs.size(); ++i) b->eng.qs_host[i].src = srcs[i];
  return engine_upload_queries(b->eng, b->stream);
}

extern "C" int adds_batch_dist_ptr(adds_batch *b, uint32_t q, void **dptr) {
  if (!b || !dptr || q >= b->srcs.size()) return ADDS_ERR_INVALID;
  *dptr = b->dist_all + b->dist_off[q];
  return ADDS_OK;
}

extern "C" int adds_batch_dist_all(adds_batch *b, void *out, uint64_t *offsets, uint64_t *total) {
  if (!b) return ADDS_ERR_INVALID;
  const size_t nq = b->srcs.size();
  const size_t tot = b->dist_off[nq - 1] + b->qgraph[nq - 1]->n;
  if (offsets)
    for (size_t q = 0; q < nq; ++q) offsets[q] = b->dist_off[q];
  if (total) *total = tot;
  if (!out) return ADDS_OK;
  CK(cudaSetDevice(b->device));
  const bool dev = is_device_ptr(out);
  CK(cudaMemcpyAsync(out, b->dist_all, tot * 4, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                     b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return ADDS_OK;
}

extern "C" int adds_batch_dist(adds_batch *b, uint32_t q, void *out) {
  if (!b || !out || q >= b->srcs.size()) return ADDS_ERR_INVALID;
  CK(cudaSetDevice(b->device));
  const bool dev = is_device_ptr(out);
  CK(cudaMemcpyAsync(out, b->dist_all + b->dist_off[q], (size_t)b->qgraph[q]->n * 4,
                     dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return ADDS_OK;
}

/* accessors used by adjoint.cu */
int adds_batch_internal(adds_batch *b, cudaStream_t *st, unsigned *nq,
                        std::vector<adds_graph *> **qgraph, std::vector<uint32_t> **srcs,
                        std::vector<adds_graph *> **ugraph, std::vector<unsigned> **qgid,
                        unsigned **dist_all, std::vector<size_t> **dist_off, void ***adj) {
  *st = b->stream;
  *nq = (unsigned)b->srcs.size();
  *qgraph = &b->qgraph;
  *srcs = &b->srcs;
  *ugraph = &b->ugraph;
  *qgid = &b->qgid;
  *dist_all = b->dist_all;
  *dist_off = &b->dist_off;
  *adj = &b->adj;
  return ADDS_OK;
}
void adds_graph_internal(const adds_graph *g, const unsigned **row, const uint2 **edges,
                         uint32_t *n, uint64_t *m, unsigned *max_deg, int *device) {
  *max_deg = g->max_deg;
  *row = g->row;
  *edges = g->edges;
  *n = g->n;
  *m = g->m;
  *device = g->device;
}

/* ------------------------------------------------------------------------ */
/* autotuner: coordinate descent over (delta, window, batch, CTAs/SM, hub
 * threshold) on the sample sources; stores the winner in the graph. */
/* device time of the sample solves: the better of two rounds after a warm
 * one (a candidate's margin is often a few percent) */
static double time_solves(adds_graph *g, const uint32_t *srcs, uint32_t ns, const adds_opts *o) {
  for (uint32_t i = 0; i < ns; ++i)
    if (adds_sssp_async(g, srcs[i], o)) return 1e30; /* warm */
  if (adds_graph_sync(g, nullptr)) return 1e30;
  cudaEvent_t a, z;
  cudaEventCreate(&a);
  cudaEventCreate(&z);
  /* three timed rounds, the median kept: the asynchronous engine's time
   * varies from run to run with its schedule (20-30 ms on the 4096^2 grid),
   * and the best of a few rounds would favour the knobs that vary most.  A
   * round during which adds_graph_sync had to regrow the worklist pool and
   * rerun the solves timed only their failed attempts, so it does not count
   * and is run again (at most twice) on the larger pool */
  double t[3] = {1e30, 1e30, 1e30};
  int counted = 0;
  for (int round = 0; counted < 3 && round < 5; ++round) {
    const unsigned grow0 = g->grow;
    cudaEventRecord(a, g->stream);
    for (uint32_t i = 0; i < ns; ++i)
      if (adds_sssp_async(g, srcs[i], o)) {
        cudaEventDestroy(a);
        cudaEventDestroy(z);
        return 1e30;
      }
    cudaEventRecord(z, g->stream);
    const int rc = adds_graph_sync(g, nullptr);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, z);
    if (rc) {
      counted = 0;
      break;
    }
    if (g->grow != grow0) continue;
    t[counted++] = ms;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(z);
  if (counted == 0) return 1e30;
  std::sort(t, t + counted);
  return t[(counted - 1) / 2];
}

extern "C" int adds_diag_wait_timeout(int device, int timeout_ms, double *waited_ms) {
  if (timeout_ms <= 0 || timeout_ms > 10000) return ADDS_ERR_INVALID;
  unsigned err = 0, where = 0;
  float ms = 0.f;
  if (ph_diag_wait(device, (unsigned)timeout_ms, &err, &where, &ms) != 0)
    return cuda_fail(cudaGetLastError(), "diagnostic wait");
  if (waited_ms) *waited_ms = ms;
  if (err == 0u) return ADDS_OK;
  snprintf(g_last_err, sizeof g_last_err, "device error %u at wait site %u", err, where);
  return err == PH_ERR_TIMEOUT ? ADDS_ERR_DEVICE_TIMEOUT : ADDS_ERR_CUDA;
}

extern "C" int adds_tune(adds_graph *g, const uint32_t *srcs, uint32_t ns, adds_opts *best,
                         double *best_ms) {
  if (!g || !srcs || ns == 0) return ADDS_ERR_INVALID;
  for (uint32_t i = 0; i < ns; ++i)
    if (srcs[i] >= g->n) return ADDS_ERR_INVALID;
  int rc = set_device(g->device);
  if (rc) return rc;
  g->tuned = 0;
  /* the defaults of one engine, every knob spelled out */
  Knobs k;
  int s0;
  float sc;
  auto defaults = [&](int engine) {
    adds_opts o;
    adds_opts_init(&o);
    o.engine = engine;
    resolve(g, &o, &k, &s0, &sc);
    o.delta_shift = s0;
    o.delta_scale = sc;
    o.window = k.window;
    o.batch_max = k.batch_max;
    o.hub_threshold = k.hub_threshold;
    o.strict_order = k.strict;
    o.local_max = k.local_max;
    o.light_heavy = k.light_heavy;
    o.block_threads = k.block;
    o.greed = k.greed;
    o.engine = k.engine;
    o.solo_max = k.solo_max;
    o.adapt = k.adapt;
    return o;
  };
  /* Coordinate descent of one engine's knobs from a start point; returns the
   * best options found and their time. */
  auto descend = [&](adds_opts cur, double bm, adds_opts *out) {
    resolve(g, &cur, &k, &s0, &sc); /* knobs of the engine */
    auto try_field = [&](int32_t adds_opts::*f, const std::vector<int> &vals) {
      for (int v : vals) {
        if (v == cur.*f) continue;
        adds_opts t = cur;
        t.*f = v;
        const double ms = time_solves(g, srcs, ns, &t);
        if (ms < bm * 0.98) {
          bm = ms;
          cur = t;
        }
      }
    };
    std::vector<int> shifts;
    for (int d = -4; d <= 4; ++d)
      if (s0 + d >= 0 && s0 + d <= 31) shifts.push_back(s0 + d);
    try_field(&adds_opts::delta_shift, shifts);
    if (cur.engine == ADDS_ENGINE_PHASE) {
      /* kernel variant (threads per CTA x CTAs per SM), then the schedule */
      const int combos[6][2] = {{256, 4}, {512, 2}, {1024, 1}, {256, 2}, {512, 1}, {128, 8}};
      for (const auto &cb : combos) {
        adds_opts t = cur;
        t.block_threads = cb[0];
        t.ctas_per_sm = cb[1];
        if (t.block_threads == cur.block_threads && t.ctas_per_sm == cur.ctas_per_sm) continue;
        const double ms = time_solves(g, srcs, ns, &t);
        if (ms < bm * 0.98) {
          bm = ms;
          cur = t;
        }
      }
      /* fewer CTAs for graphs whose phases are too short to use the GPU */
      if (g->m < (1ull << 24)) try_field(&adds_opts::group_ctas, {8, 16, 32, 64, 148});
      try_field(&adds_opts::solo_max, {0, 256, 512, 1024, 2048, 4096, 16384});
      try_field(&adds_opts::hub_threshold, {128, 256, 1024, 4096});
      try_field(&adds_opts::light_heavy, {0, 1, 2});
      try_field(&adds_opts::adapt, {0, 1});
      /* 3: after a pull phase, the next bucket's list is mostly stale entries
       * (R-MAT 24: 4.41 against 4.55 ms with dense_scan off) */
      try_field(&adds_opts::dense_scan, {3, 4, 6, 8});
    } else {
      try_field(&adds_opts::window, {1, 2, 3, 4, 8});
      try_field(&adds_opts::batch_max, {64, 128, 256, 512});
      try_field(&adds_opts::hub_threshold, {4096, 16384, 65536});
      try_field(&adds_opts::block_threads, {128, 256, 512});
      try_field(&adds_opts::greed, {0, 2, 4, 8});
      int maxb = g->eng.max_bps[block_index(cur.block_threads > 0 ? cur.block_threads : 256)];
      std::vector<int> cps;
      for (int c = 1; c <= maxb; ++c) cps.push_back(c);
      try_field(&adds_opts::ctas_per_sm, cps);
      try_field(&adds_opts::strict_order, {0, 1});
      try_field(&adds_opts::local_max, {0, 64, 256, 512});
      try_field(&adds_opts::light_heavy, {0, 1});
      try_field(&adds_opts::adapt, {0, 1});
    }
    if (cur.delta_shift != s0) { /* second look around the new delta */
      std::vector<int> s2;
      for (int d = -1; d <= 1; ++d)
        if (cur.delta_shift + d >= 0 && cur.delta_shift + d <= 31) s2.push_back(cur.delta_shift + d);
      try_field(&adds_opts::delta_shift, s2);
    }
    *out = cur;
    return bm;
  };
  /* in: the engine to tune; auto times both and tunes the faster one (the
   * phase engine wins on low-diameter graphs, the asynchronous one where
   * thousands of buckets each hold a thin frontier).  Small graphs (under
   * 2^24 edges, where a solve takes well under a millisecond) get a full
   * descent of both engines, since a start point does not predict the
   * winner there (the phase engine on few CTAs needs its knobs first). */
  const int want = (best && best->engine > 0) ? best->engine : ADDS_ENGINE_AUTO;
  adds_opts cur = defaults(want == ADDS_ENGINE_ASYNC ? ADDS_ENGINE_ASYNC : ADDS_ENGINE_PHASE);
  double bm = time_solves(g, srcs, ns, &cur);
  if (want == ADDS_ENGINE_AUTO && g->m < (1ull << 24)) {
    adds_opts bp, ba;
    adds_opts p0 = cur;
    p0.group_ctas = 32;
    const double m0 = time_solves(g, srcs, ns, &p0);
    const double mp = descend(m0 < bm ? p0 : cur, m0 < bm ? m0 : bm, &bp);
    const adds_opts a0 = defaults(ADDS_ENGINE_ASYNC);
    const double ma = descend(a0, time_solves(g, srcs, ns, &a0), &ba);
    cur = mp <= ma ? bp : ba;
    bm = mp <= ma ? mp : ma;
  } else {
    if (want == ADDS_ENGINE_AUTO) {
      const adds_opts alt = defaults(ADDS_ENGINE_ASYNC);
      const double ma = time_solves(g, srcs, ns, &alt);
      if (ma < bm) {
        bm = ma;
        cur = alt;
      }
    }
    bm = descend(cur, bm, &cur);
  }
  if (bm >= 1e29) return ADDS_ERR_DEVICE_TIMEOUT;
  /* the wave kernels, on the width that an untuned solve gives them (they adapt
   * it); the winner is kept as it was timed, beside the engine's knobs */
  adds_opts won;
  adds_opts_init(&won);
  if (want == ADDS_ENGINE_AUTO && g->m < (1ull << 31)) {
    for (int v = 0; v <= WV_LAST; ++v) {
      adds_opts w;
      adds_opts_init(&w);
      w.engine = ADDS_ENGINE_PHASE;
      w.wave = v + 1;
      w.delta_shift = v == WV_POOL ? pooled_shift(g, auto_shift(g)) : auto_shift(g);
      w.delta_scale = auto_scale(g);
      g->wave_off = false;
      const double ms = time_solves(g, srcs, ns, &w);
      if (!g->wave_off && ms < bm * 0.98) { /* off: its lists overflowed */
        bm = ms;
        won = w;
      }
    }
    g->wave_off = false;
    if (won.wave == 0) wv_engine_free(g->weng); /* the lists of the last trial */
  }
  g->tuned_opts = cur;
  g->tuned_opts.stream = nullptr;
  g->tuned_wave = won;
  g->tuned = 1;
  if (best) *best = won.wave > 0 ? won : g->tuned_opts;
  if (best_ms) *best_ms = bm / ns;
  return ADDS_OK;
}
