// Forward kernels of the spiking substrate: LIF integration over the CSR
// graph with integer delays in a delay ring and event-driven delivery.
//
// Reference semantics: run_cpu, src/runtime/cpu_backend.cpp:67-191 (serial
// branch).  Per step t of one sample:
//   ext[i]   = drive of step t summed in event order        (:99)
//   if refr: refr--, v = reset                              (:130-132)
//   else     v = v*decay + ext + ring[t%R][i]; fire if v >= thr  (:134-139)
//   ring[t%R][i] = 0                                         (:142)
//   logits[channel] += 1 for fired OUTPUT neurons           (:149-151)
//   for fired i in ascending id, for e in row(i) in order:
//            ring[(t+d_e)%R][post_e] += sign_i * w_e         (:173-181)
//
// Three kernel families share the per-step phases below:
//   tier S  (k_tier_s)  one CTA simulates one sample with its whole state
//           and delay ring in shared memory; CTAs pull samples from a work
//           queue (longest first), so uneven step counts balance across SMs.
//   tier G  (k_tier_g)  every SM cooperates on a wave of samples in lockstep;
//           CTA b owns neuron block b: its v / refr and (SORT, BUCKET) its
//           ring columns live in shared memory for the whole launch, and a
//           bounded software grid barrier separates the two phases of a step.
//   plain   (k_plain_a / k_plain_b) the same phases as one kernel launch
//           each per step with state in global memory, one sample after
//           another: the per-sample path.
//
// Delivery modes (include/snc_b200.h):
//   ATOMIC  the owner of a fired neuron adds its row into the global ring
//           with red.add (one barrier per step).
//   BUCKET  the owner of a fired neuron posts one (first edge, length)
//           descriptor per destination block to that block's inbox; after the
//           barrier each block expands its inbox and accumulates into its
//           shared-memory ring slice with shared atomics.
//   SORT    as BUCKET, but every ring cell receives its contributions in
//           (pre, edge) order -- per-cell lists in a shared hash table, each
//           ordered by gedges index or staging order: the result is
//           bit-identical to the serial CPU backend.
#include <algorithm>
#include <climits>
#include <cstring>
#include <initializer_list>

#include "device_common.cuh"
#include "internal.h"

namespace sncb {

enum { MODE_ATOMIC = 0, MODE_BUCKET = 1, MODE_SORT = 2 };

constexpr int kGThreads = 512;      // plain-path block size; tier G minimum
constexpr int kGThreadsMax = 768;   // tier G block size bound (one CTA per SM)
constexpr int kGChunk = 1024;       // staged events per ordered-apply chunk
constexpr int kGDesc = 1024;        // inbox descriptors handled per chunk
constexpr int kMaxWave = 64;        // samples per lockstep wave

struct FwdArgs {
  // graph
  int N, S, R, ncols, noc, P, BS, G;
  const int* row_ptr;
  const uint2* edges;
  const uint2* gedges;
  const int* gptr;
  const int2* groups;
  const int* col_of;
  const int* out_ch;
  const int* colbase;
  const int* ibase;
  // inputs
  int B;
  const int* order;
  const int* steps;
  const long long* sptr_off;
  const long long* stepbase;
  const int* sched_ptr;
  const int* sched_nid;
  const float* sched_ext;
  const int* sched_blk;  // [total_steps][P+1] or null
  const long long* raster_off;
  // outputs
  int* counts;
  unsigned long long* spikes;
  unsigned long long* events;
  uint32_t* raster;
  float* vfinal;
  int W;
  // grid / plain state
  int Bw;
  float* v;
  int* refr;
  float* ring;
  int* fired;
  int* fired_cnt;
  unsigned long long* inbox;  // [Bw][2][G]
  int* inbox_cnt;             // [Bw][2][P]
  // control
  int* err;
  unsigned* ctl;
  LifP lif;
  // e-prop (tier S only): eligibility [B][S], per-neuron fire counts
  float* elig;
  unsigned long long* fires;
  float gamma, trace_decay;
  // tier S: edges with each row regrouped by column range, (delay * ncols +
  // column, weight), and the segment starts [N][kSPtr]; fired rows whose
  // segment starts shared memory holds at once; mask of the conflict tags
  const uint2* sedges;
  const int* sptr;
  int s_cap;
  int s_tmask;
  // ring columns of a CTA and the neurons' (the CTA's part of a cluster's)
  int s_nc;
  const int* s_col;
  // deferred eligibility: psi of every ring column and step, [B][ncols][psi_T]
  // (null: eligibility accumulated in the forward into elig)
  float* psi_hist;
  int psi_T;
  // tier G: groups of threads that take a wave's samples side by side (1: the
  // whole CTA one after another)
  int g_groups, g_threads;
  // bound of the grid barrier's waits (0: the default) and arrivals that no
  // block makes (a stall injected for failure tests: every wait runs out)
  unsigned long long wait_ns;
  unsigned stall;
  // leaky readout units (ro_on): OUTPUT neurons integrate v = ro_decay * v +
  // drive + ring and never fire; each sample's final potentials go to
  // ro_v [B][n_ro] at their rank, k_readout_logits turns them into logits
  int ro_on;
  float ro_decay;
  const int* ro_rank;
  const int* ro_chan;
  int n_ro;
  float* ro_v;
  float* ro_logits;
  // post-neuron partitions (plain kernels only): first neuron block of the
  // grid, no inbox descriptors posted, delivery by scanning every block's
  // fired list (SORT)
  int blk0;
  int no_post;
  int scan_only;
};

// Shared memory that decides whether a sample's state fits one CTA (tier S).
// The kernel itself never needs more (tier_s_layout below).
static size_t tier_s_bytes(int N, int ncols, int R, int noc, int mode, bool eprop, int nthr) {
  size_t words = (size_t)R * ncols + 4 * (size_t)N + (size_t)noc;
  if (mode == MODE_SORT) words += (size_t)N + 1 + 2 * (size_t)ncols + 4 * (size_t)nthr;
  if (eprop) words += (size_t)N + ncols;
  return words * 4 + 16;
}

int tier_s_smem_bytes(const Graph* g, int mode, bool eprop) {
  return (int)tier_s_bytes(g->N, g->ncols, g->R, std::max(1, g->noc), mode, eprop, 1024);
}

// ---------------------------------------------------------------------------
// one LIF neuron (cpu_backend.cpp:129-143, plus reset_mode 1 = subtractive)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int lif_step(const LifP& p, float& v, int& refr, float ext, float rin,
                                        float* vpre = nullptr) {
  // without branches: the refractory and the integrating neurons of a warp
  // together
  const bool idle = refr > 0;
  const float nv = lif_integrate(v, p.decay, ext, rin);
  if (vpre) *vpre = idle ? p.reset : nv;
  const bool f = !idle && nv >= p.thr;
  const float vf = p.reset_mode ? __fsub_rn(nv, p.thr) : p.reset;
  v = idle ? p.reset : f ? vf : nv;
  refr = idle ? refr - 1 : f ? p.refractory : refr;
  return f;
}

// A leaky readout unit (shd_model.py:139-140 with the substrate's delivered
// current as its input): v = ro_decay * v + ext + ring, rounded like the LIF
// integration; it never fires or resets.
__device__ __forceinline__ int readout_step(float ro_decay, float& v, float ext, float rin,
                                            float* vpre = nullptr) {
  v = lif_integrate(v, ro_decay, ext, rin);
  if (vpre) *vpre = v;
  return 0;
}

// logits[b][c] = sum over the readout units of channel c, ascending id, of
// their final potential / T_b (shd_model.py:147 averages the readout over
// the steps).  One block per sample, a thread per channel.
__global__ void k_readout_logits(const float* __restrict__ ro_v, const int* __restrict__ ro_chan,
                                 int n_ro, const int* __restrict__ steps, int noc,
                                 float* __restrict__ logits) {
  const int b = blockIdx.x;
  const float T = (float)max(1, steps[b]);
  for (int c = threadIdx.x; c < noc; c += blockDim.x) {
    float acc = 0.f;
    for (int r = 0; r < n_ro; ++r)
      if (ro_chan[r] == c) acc = __fadd_rn(acc, __fdiv_rn(ro_v[(size_t)b * n_ro + r], T));
    logits[(size_t)b * noc + c] = acc;
  }
}

// Ring slot of a delivery made at step slot `s0` with delay d (1 <= d < R).
__device__ __forceinline__ int ring_slot(int s0, int d, int R) {
  const int s = s0 + d;
  return s >= R ? s - R : s;
}

template <bool GLOBAL_RING>
__device__ __forceinline__ void apply_one(float* ring, int ring_stride, int col0, int c, int slot,
                                          float w) {
  float* cell = ring + (size_t)slot * ring_stride + col0 + c;
  if (GLOBAL_RING) {
    __stcg(cell, __fadd_rn(__ldcg(cell), w));
  } else {
    *cell = __fadd_rn(*cell, w);
  }
}

// Chunks up to kCountMax events take the per-cell apply; larger ones are
// linked in order (a post block owns hub columns whose per-step event count can
// be large).
constexpr int kCountMax = 256;
constexpr int kFirstFlag = 1 << 30;  // marks a group's first event of its column in st_col

// Ordered apply of a small chunk (ce <= kCountMax <= blockDim.x, so thread q
// owns staged event q) through its ring cells.  A hash table of kCellTable
// keys (column, slot) -- zeroed by the caller before staging -- holds one
// unordered list per cell (atomicExch heads, one link per event).  The first
// arrival at a cell owns it: alone there, it applies its event; otherwise it
// collects the cell's list (kCellSort entries in registers, sorted; longer
// lists by repeated minimum selection) and applies it in order.  A step's
// events spread over many more cells than columns -- a column's events carry
// different delays -- so lists are short and no thread walks a hub column's
// whole chain.
constexpr int kCellTable = 2 * kCountMax;  // keys, then list heads (q + 1, 0 = empty)
constexpr int kCellSort = 8;
static_assert(2 * kCellTable <= kGChunk, "the table lives in st_next");
static_assert(kCellTable + kCountMax <= kGChunk, "the links live in st_col beyond the chunk");

// Table sizes (keys; as many list heads follow) and their hash bits.
template <int TS>
constexpr int kTabBits = TS == 1024 ? 10 : 9;

// Enters staged event q of cell (c, sl) into a table of TS keys (at most TS / 2
// distinct cells); returns its entry.
template <int TS>
__device__ __forceinline__ unsigned cell_insert(int* tab, int* link, int q, int c, int sl, bool* first) {
  static_assert(TS == 512 || TS == 1024, "table size");
  unsigned* key = reinterpret_cast<unsigned*>(tab);
  const unsigned k = (unsigned)c * 256u + (unsigned)sl + 1u;  // slot < 256, 0 = empty
  unsigned h = (k * 2654435761u) >> (32 - kTabBits<TS>);
  // at most TS / 2 keys: a free or equal entry is always found
  for (int probe = 0; probe < TS; ++probe) {
    const unsigned old = atomicCAS(&key[h], 0u, k);
    if (old == 0u || old == k) break;
    h = (h + 1u) & (TS - 1);
  }
  const int prev = atomicExch(&tab[TS + h], q + 1);
  link[q] = prev;
  *first = prev == 0;
  return h;
}

// The owner's part (after a barrier that follows every cell_insert): apply
// the cell's events in increasing order -- their staging index, or with
// KEYED their order key okey[x] (unique per event) -- then x.
template <bool GLOBAL_RING, bool KEYED>
__device__ __forceinline__ void cell_apply_list(int top, const int* link, const int* okey,
                                                const float* st_w, int q, int c, int sl, float* ring,
                                                int ring_stride, int col0) {
  if (top == q + 1) {
    apply_one<GLOBAL_RING>(ring, ring_stride, col0, c, sl, st_w[q]);
    return;
  }
  auto ord = [&](int x) -> long long {
    return KEYED ? ((long long)okey[x] << 10) | x : (long long)x;  // x < kGChunk = 1024
  };
  long long r[kCellSort];
#pragma unroll
  for (int i = 0; i < kCellSort; ++i) r[i] = LLONG_MAX;
  int p = top;
#pragma unroll
  for (int i = 0; i < kCellSort; ++i) {
    if (p != 0) {
      // insert into the sorted r (its largest entry is free)
      r[kCellSort - 1] = ord(p - 1);
#pragma unroll
      for (int m = kCellSort - 1; m > 0; --m) {
        const long long lo = min(r[m - 1], r[m]), hi = max(r[m - 1], r[m]);
        r[m - 1] = lo;
        r[m] = hi;
      }
      p = link[p - 1];
    }
  }
  if (p == 0) {
#pragma unroll
    for (int i = 0; i < kCellSort; ++i)
      if (r[i] != LLONG_MAX) apply_one<GLOBAL_RING>(ring, ring_stride, col0, c, sl, st_w[(int)(r[i] & 1023)]);
    return;
  }
  long long last = -1;
  for (;;) {
    long long best = LLONG_MAX;
    for (int x = top; x != 0; x = link[x - 1]) {
      const long long o = ord(x - 1);
      if (o > last && o < best) best = o;
    }
    if (best == LLONG_MAX) break;
    apply_one<GLOBAL_RING>(ring, ring_stride, col0, c, sl, st_w[(int)(best & 1023)]);
    last = best;
  }
}

template <bool GLOBAL_RING, bool KEYED, int TS>
__device__ __forceinline__ void cell_apply(const int* tab, const int* link, const int* okey,
                                           const float* st_w, unsigned h, int q, int c, int sl,
                                           float* ring, int ring_stride, int col0) {
  cell_apply_list<GLOBAL_RING, KEYED>(tab[TS + h], link, okey, st_w, q, c, sl, ring, ring_stride, col0);
}

template <bool GLOBAL_RING, class G>
__device__ void apply_cells(const G& grp, int ce, int* tab, int* st_col, const int* st_slot, const float* st_w,
                            float* ring, int ring_stride, int col0) {
  int* link = st_col + kCellTable;
  const int q = grp.tid();
  int c = 0, sl = 0;
  unsigned h = 0;
  bool first = false;
  if (q < ce) {
    c = st_col[q];
    sl = st_slot[q];
    h = cell_insert<kCellTable>(tab, link, q, c, sl, &first);
  }
  grp.sync();
  if (first)
    cell_apply<GLOBAL_RING, false, kCellTable>(tab, link, nullptr, st_w, h, q, c, sl, ring, ring_stride,
                                               col0);
  grp.sync();
}

// Ordered apply of one chunk of staged events.  Staging index q is the
// (pre, edge) order of the CPU backend.  The events were staged with their
// block-local column st_col[q] (head / tail of every local column = -1).
// Every ring cell must receive its contributions in increasing q.
//  - chunks up to kCountMax events: apply_cells (above);
//  - larger chunks: every warp links the events of its 32-event groups
//    (match.any: successor within the group, first event of each column
//    flagged), then one warp joins the groups in staging order through the
//    column tails -- one shared-memory round trip per group; one thread per
//    column then replays its list: O(events), no sorting, and hub columns
//    with many events in one step stay linear.
template <bool GLOBAL_RING, class G>
__device__ void apply_ordered(const G& grp, int ce, int* head, int* tail, int ncols_local, int* st_col,
                              const int* st_slot, const float* st_w, int* st_next, float* ring,
                              int ring_stride, int col0) {
  grp.sync();
  if (ce <= kCountMax && ce <= (int)grp.size()) {
    apply_cells<GLOBAL_RING>(grp, ce, st_next, st_col, st_slot, st_w, ring, ring_stride, col0);
    return;
  }
  {
    // 1. every warp links its own 32-event groups (match.any): successor
    //    within the group or -1, first event of each column flagged
    const int lane = grp.tid() & 31, warp = grp.tid() >> 5, nwarps = grp.size() >> 5;
    const unsigned below = (1u << lane) - 1u;
    for (int g0 = warp * 32; g0 < ce; g0 += nwarps * 32) {
      const int q = g0 + lane;
      const bool valid = q < ce;
      const int c = valid ? st_col[q] : -1 - lane;
      const unsigned peers = __match_any_sync(0xffffffffu, c);
      const unsigned higher = peers & ~below & ~(1u << lane);
      if (valid) {
        st_next[q] = higher ? g0 + __ffs(higher) - 1 : -1;
        if (!(peers & below)) st_col[q] = c | kFirstFlag;
      }
    }
  }
  grp.sync();
  // 2. one warp joins the groups in order through the column tails
  if (grp.tid() < 32) {
    const int lane = grp.tid();
    for (int g0 = 0; g0 < ce; g0 += 32) {
      const int q = g0 + lane;
      int c = 0, t = -1;
      bool first = false, last = false;
      if (q < ce) {
        const int cf = st_col[q];
        first = (cf & kFirstFlag) != 0;
        c = cf & ~kFirstFlag;
        last = st_next[q] < 0;
        if (first) t = tail[c];
      }
      __syncwarp();
      if (first) {
        if (t >= 0) st_next[t] = q;
        else head[c] = q;
      }
      if (last) tail[c] = q;
      __syncwarp();
    }
  }
  grp.sync();
  for (int c = grp.tid(); c < ncols_local; c += grp.size()) {
    int p = head[c];
    if (p < 0) continue;
    head[c] = -1;
    tail[c] = -1;
    for (; p >= 0; p = st_next[p]) apply_one<GLOBAL_RING>(ring, ring_stride, col0, c, st_slot[p], st_w[p]);
  }
  grp.sync();
}

constexpr int kSThreads = 1024;
// deliveries of the tier-S kernel (kSRoom: ordered, fewer than 128 rows staged)
enum { kSAtomic = 0, kSOrdered = 1, kSRoom = 2 };
constexpr int kSRows = 4;   // fired rows of a lane: a tier-S warp takes 128 at once
constexpr int kSAhead = 2;  // 32-event groups whose edges a tier-S warp keeps in flight
// ints of scratch of a tier-S warp that stages up to cap rows
__host__ __device__ constexpr int s_scratch(int cap) { return (cap < 32 * kSRows ? cap : 32 * kSRows) + 32 + 4; }
constexpr int kSOff = kSPtr + 1;  // ints of a staged row (odd: no bank conflicts)

// Barrier of the thread-block cluster; orders shared-memory writes of its CTAs
// to one another.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// *p = v in CTA `rank` of the cluster (p: this CTA's address of the same place).
__device__ __forceinline__ void st_cluster(int* p, int rank, int v) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(r), "r"(v) : "memory");
}

__device__ __forceinline__ int lds_i(unsigned a) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float lds_f(unsigned a) { return __int_as_float(lds_i(a)); }
__device__ __forceinline__ int lds_b(unsigned a) {
  int v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_i(unsigned a, int v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_f(unsigned a, float v) { sts_i(a, __float_as_int(v)); }
__device__ __forceinline__ void sts_b(unsigned a, int v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Copies the segment starts of row j (and the end of its last segment) to
// shared memory, asynchronously (the whole warp; cp.async.wait_all follows).
__device__ __forceinline__ void stage_row(const int* __restrict__ sptr, int j, int* dst, int lane) {
  static_assert(kSPtr == 32, "an entry per lane");
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst + lane)),
               "l"(sptr + j * kSPtr + lane)
               : "memory");
}

// ---------------------------------------------------------------------------
// tier S: one CTA per sample, state in registers and shared memory
// ---------------------------------------------------------------------------
// Every warp owns a set of the ring's columns (kSRanges ranges of about equal
// in-degree, hub columns spread over them) and is the only one that ever adds to their cells, so
// the delivery of a step needs no barrier, no float atomics and no tables: the
// warp walks the step's fired rows in ascending order, reads its own segment
// of each row (sedges: the row stably regrouped by range; sptr: the segment
// starts), 32 events at a time, and adds them.  Events of one 32-event group
// that meet in a cell are added one after another in lane order; every other
// pair of a cell's events is in program order.  That is the CPU backend's
// (pre, edge) order: SORT, bit for bit.
//
// CL > 1: a cluster of CL CTAs per sample, each with every CL-th word of 32
// neurons and their columns.  They exchange the fired bits of a step through
// distributed shared memory before the cluster barrier that takes the place of
// the first CTA barrier; everything after it is the CTA's own.
//
// What bounds it, on a 1744-neuron net (197 k synapses, delays to 30) at 57
// fired rows and 7000 events a step, in cycles of a step (15,000): integration
// 2600, list and the copy of the segment starts 1400 and 900 (L2), a warp's
// segments 2300, its first edges 600 (L2), 7 groups of 32 events a warp 7500 --
// eight warps a scheduler, two thirds of a group shared-memory passes over
// random cells (tag, ring).  7.5 us a step, 17.2 with events staged 1024 at a
// time by a search per event and ordered through cell bitmaps and a hash table;
// ATOMIC 4.0 us, 6.0 with the rows of a warp's list fetched one after another;
// a 1050-neuron net with 90 short rows a step 4.2 us, 5.2 before.  Clusters of
// four: 5.8 us for up to 33 samples.  Slower: 16 ranges and warps (too few in
// flight), owners that add one row's segment at a time without a conflict check
// (130 cycles a row for the chain), match.any for the conflicts (100 cycles a
// group), edges requested 4 or 8 groups ahead in registers (they share
// scoreboards, so the oldest waits for the newest).
template <int KN, bool EP, int DEL, int CL>
__global__ void __launch_bounds__(kSThreads, 1) k_tier_s(FwdArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long lscratch[40];
  __shared__ int s_q;
  constexpr int nthr = kSThreads, nwarps = nthr / 32;
  // ring columns of this CTA (all of them, or its part of a cluster's)
  const int N = a.N, R = a.R, nc = a.s_nc, noc = a.noc, RN = R * nc;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int nch = KN ? KN : (N + nthr - 1) / nthr;  // neurons of a thread
  const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0, nwords = (N + 31) >> 5;
  // the 32 neurons of this warp's chunk c
  auto word_of = [&](int c) { return CL > 1 ? (c * nwarps + warp) * CL + rank : c * nwarps + warp; };
  float* ring = reinterpret_cast<float*>(smem_raw);
  float* ext = ring + RN;
  int* counts = reinterpret_cast<int*>(ext + N);
  // [nch][nwarps] fired neurons of each 32; cluster: [2][nwords] fired bits of
  // all neurons, steps alternating
  int* wcnt = counts + noc;
  float* sv = reinterpret_cast<float*>(wcnt + (CL > 1 ? 2 * nwords : nch * nwarps));  // KN == 0 only
  int* srefr = reinterpret_cast<int*>(sv + (KN ? 0 : N));
  float* tr = reinterpret_cast<float*>(srefr + (KN ? 0 : N));  // inline eligibility only
  const bool inl = EP && a.elig;
  float* psi = tr + (inl ? N : 0);
  int* off = reinterpret_cast<int*>(psi + (inl ? nc : 0));  // [s_cap][kSOff] staged rows
  // per warp: segment offsets and segment marks.
  int* scr0 = off + (DEL == kSAtomic ? 0 : a.s_cap * kSOff);
  // 128 rows' segments and then the marks, at constant places, where that measured
  // faster (70 samples of a 998-neuron net 494 us, 504 in the other order); else
  // the marks first and as many segments as are staged
  constexpr bool kFull = DEL == kSOrdered && KN == 1 && (!EP || CL > 1);
  const int n_scr = s_scratch(kFull ? 32 * kSRows : a.s_cap);
  unsigned* mark = reinterpret_cast<unsigned*>(scr0 + (DEL == kSAtomic ? 0 : warp * n_scr) + (kFull ? 32 * kSRows : 0));
  unsigned short* fired = reinterpret_cast<unsigned short*>(scr0 + (DEL == kSAtomic ? 0 : nwarps * n_scr));
  // a byte per cell, or s_tmask + 1 per warp
  unsigned char* tag = reinterpret_cast<unsigned char*>(fired + N) + (a.s_tmask == INT_MAX ? 0 : warp * (a.s_tmask + 1));
  const int tmask = a.s_tmask;
  const LifP lif = a.lif;
  const float thr = lif.thr;
  // the delivery's arrays as shared addresses
  const unsigned ring_s = (unsigned)__cvta_generic_to_shared(ring);
  const unsigned off_w = (unsigned)__cvta_generic_to_shared(off + lane * kSOff + warp);
  const unsigned mark_s = (unsigned)__cvta_generic_to_shared(mark);
  const unsigned scr_s = kFull ? mark_s - 4 * 32 * kSRows : mark_s + 4 * 36;
  const unsigned tag_s = (unsigned)__cvta_generic_to_shared(tag);
  const unsigned upto = below | (1u << lane);
  const uint2* __restrict__ sed = a.sedges;

  float vr[KN ? KN : 1];
  int rf[KN ? KN : 1], colr[KN ? KN : 1], colg[EP && CL > 1 && KN ? KN : 1];  // colg: in the graph
  unsigned outm = 0;  // bit c: the neuron is an output with a channel
#pragma unroll
  for (int c = 0; c < nch; ++c) {
    const int j = 32 * word_of(c) + lane;
    if (KN) colr[KN ? c : 0] = j < N ? a.s_col[j] : -1;
    if (EP && CL > 1) colg[EP && CL > 1 && KN ? c : 0] = j < N ? a.col_of[j] : -1;
    if (j < N && a.out_ch[j] >= 0) outm |= 1u << c;
  }
  const unsigned rom = a.ro_on ? outm : 0u;  // bit c: a leaky readout unit

  for (int round = 0;; ++round) {
    int q;
    if (CL > 1) {  // a cluster per sample
      q = round ? a.B : (int)(blockIdx.x / CL);
    } else {
      if (tid == 0) s_q = (int)atomicAdd(&a.ctl[1], 1u);
      __syncthreads();
      q = s_q;
    }
    if (q >= a.B) break;
    const int b = a.order[q];
    const int T = a.steps[b];
    for (int i = tid; i < RN; i += nthr) ring[i] = 0.f;
    for (int i = tid; i < N; i += nthr) {
      ext[i] = 0.f;
      if (!KN) {
        sv[i] = 0.f;
        srefr[i] = 0;
      }
      if (inl) tr[i] = 0.f;
    }
    if (KN) {
#pragma unroll
      for (int c = 0; c < KN; ++c) {
        vr[c] = 0.f;
        rf[c] = 0;
      }
    }
    for (int i = tid; i < noc; i += nthr) counts[i] = 0;
    if (CL > 1) cluster_sync();  // every CTA of the cluster runs from here on
    else __syncthreads();
    const int* sp = a.sched_ptr + a.sptr_off[b];
    uint32_t* rast = a.raster ? a.raster + a.raster_off[b] : nullptr;
    float* psi_t = EP && a.psi_hist ? a.psi_hist + (size_t)b * a.psi_T * a.ncols : nullptr;
    long long n_spikes = 0, n_events = 0;  // of the sample / of this warp's columns
    int s0n = 0;                           // first cell of the current slot
    // the drive: a step's entries name distinct neurons; thread i holds entry
    // i of the next step's in registers, loaded a step ahead from a range
    // whose end was itself loaded a step earlier (entries beyond blockDim.x
    // are read when they are stored)
    int p_lo = 0, p_hi = 0, p_nx = 0, pf_nid = -1;
    float pf_ext = 0.f;
    auto fetch_drive = [&]() {
      pf_nid = -1;
      if (p_lo + tid < p_hi) {
        pf_nid = a.sched_nid[p_lo + tid];
        pf_ext = a.sched_ext[p_lo + tid];
      }
    };
    auto store_drive = [&]() {
      if (pf_nid >= 0) ext[pf_nid] = pf_ext;
      for (int k = p_lo + nthr + tid; k < p_hi; k += nthr) ext[a.sched_nid[k]] = a.sched_ext[k];
    };
    if (T > 0) {
      p_lo = sp[0];
      p_hi = sp[1];
      fetch_drive();
      store_drive();
      p_lo = p_hi;
      p_hi = sp[min(2, T)];
      fetch_drive();  // step 1
      p_nx = sp[min(3, T)];
      __syncthreads();
    }
    for (int t = 0; t < T; ++t) {
      unsigned fm = 0;  // bit c: this thread's neuron of chunk c fired
#pragma unroll
      for (int c = 0; c < nch; ++c) {
        const int wd = word_of(c), j = 32 * wd + lane;
        bool f = false;
        if (j < N) {
          float vv = KN ? vr[KN ? c : 0] : sv[j];
          int rr = KN ? rf[KN ? c : 0] : srefr[j];
          const int col = KN ? colr[KN ? c : 0] : a.s_col[j];
          const float e = ext[j];
          ext[j] = 0.f;
          float rin = 0.f;
          if (col >= 0) {
            rin = ring[s0n + col];
            ring[s0n + col] = 0.f;
          }
          // lif_step / readout_step without branches
          const bool ro = (rom >> c) & 1u, idle = !ro && rr > 0;
          const float nv = lif_integrate(vv, ro ? a.ro_decay : lif.decay, e, rin);
          f = !ro && !idle && nv >= thr;
          const float vf = lif.reset_mode ? __fsub_rn(nv, thr) : lif.reset;
          vv = idle ? lif.reset : f ? vf : nv;
          rr = idle ? rr - 1 : f ? lif.refractory : rr;
          if (KN) {
            vr[KN ? c : 0] = vv;
            rf[KN ? c : 0] = rr;
          } else {
            sv[j] = vv;
            srefr[j] = rr;
          }
          if (EP) {
            // cuda_trainer.cu:93-95: triangular surrogate and pre trace
            if (col >= 0) {
              float dd = fabsf(__fsub_rn(idle ? lif.reset : nv, thr));
              if (thr > 0.f && thr != 1.f) dd = __fdiv_rn(dd, thr);  // x / 1 = x
              const float ps = dd < 1.f ? __fmul_rn(a.gamma, __fsub_rn(1.f, dd)) : 0.f;
              if (inl) psi[col] = ps;
              if (psi_t) psi_t[EP && CL > 1 ? colg[EP && CL > 1 && KN ? c : 0] : col] = ps;
            }
            if (inl)
              tr[j] = __fadd_rn(__fmul_rn(a.trace_decay, tr[j]),
                                __fmul_rn(__fsub_rn(1.f, a.trace_decay), f ? 1.f : 0.f));
            if (f && a.fires) atomicAdd(&a.fires[j], 1ull);
          }
          if (f) {
            fm |= 1u << c;
            if ((outm >> c) & 1u) atomicAdd(&counts[a.out_ch[j]], 1);
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (CL > 1) {
          if (lane < CL && wd < nwords) st_cluster(wcnt + (t & 1) * nwords + wd, lane, (int)m);
        } else if (lane == 0) {
          wcnt[c * nwarps + warp] = __popc(m);
        }
        if (rast && lane == 0 && wd < nwords) rast[wd] = m;
      }
      if (rast) rast += a.W;
      if (EP && psi_t) psi_t += a.ncols;
      if (CL > 1) cluster_sync();
      else __syncthreads();
      // ascending fired list; the segment starts of the first s_cap fired rows
      int nf = 0;
      if (CL > 1) {
        // (at most 4 x 32 words: a cluster's threads hold every neuron)
        const unsigned* fw = reinterpret_cast<const unsigned*>(wcnt + (t & 1) * nwords);
        unsigned fwl[CL];
        int all = 0;
#pragma unroll
        for (int i = 0; i < CL; ++i) {
          fwl[i] = 32 * i + lane < nwords ? fw[32 * i + lane] : 0u;
          all += __popc(fwl[i]);
        }
        nf = __reduce_add_sync(0xffffffffu, all);
#pragma unroll
        for (int i = 0; i < CL; ++i) {
          const int wd = 32 * i + warp;
          unsigned m = __shfl_sync(0xffffffffu, fwl[i], warp);
          if (!m) continue;
          int n = 0;  // fired before word wd
#pragma unroll
          for (int k = 0; k < CL; ++k)
            if (32 * k + lane < wd) n += __popc(fwl[k]);
          int rk = __reduce_add_sync(0xffffffffu, n);
          if ((m >> lane) & 1u) fired[rk + __popc(m & below)] = (unsigned short)(32 * wd + lane);
          for (; m && rk < a.s_cap; m &= m - 1u, ++rk)
            stage_row(a.sptr, (32 * wd + __ffs(m) - 1) * CL + rank, off + rk * kSOff, lane);
        }
      } else {
#pragma unroll
        for (int c = 0; c < nch; ++c) {
          // (fired of the chunk's earlier warps, fired of the chunk) in one sum
          const int n = lane < nwarps ? wcnt[c * nwarps + lane] : 0;
          const unsigned both =
              __reduce_add_sync(0xffffffffu, (unsigned)((lane < warp ? n : 0) | (n << 16)));
          int rk = nf + (int)(both & 0xffffu);
          nf += (int)(both >> 16);
          const bool f = (fm >> c) & 1u;
          unsigned m = __ballot_sync(0xffffffffu, f);
          if (!m) continue;
          if (f) fired[rk + __popc(m & below)] = (unsigned short)(c * nthr + tid);
          if (DEL != kSAtomic)
            for (; m && rk < a.s_cap; m &= m - 1u, ++rk)
              stage_row(a.sptr, c * nthr + warp * 32 + __ffs(m) - 1, off + rk * kSOff, lane);
        }
      }
      n_spikes += nf;
      store_drive();
      p_lo = p_hi;
      p_hi = p_nx;
      fetch_drive();
      p_nx = sp[min(t + 4, T)];
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (inl) {
        // cuda_trainer.cu:105-112: E[b,s] += psi[post] * tr[pre]; rows whose
        // trace is exactly zero add +0 and are skipped (trainer.cpp:243-244)
        float* Eb = a.elig + (size_t)b * a.S;
        for (int i = warp; i < N; i += nwarps) {
          const float tri = tr[i];
          if (tri == 0.f) continue;
          const int rs = a.row_ptr[i], re = a.row_ptr[i + 1];
          for (int e = rs + lane; e < re; e += 32) {
            const uint2 ed = a.edges[e];
            Eb[e] = __fadd_rn(Eb[e], __fmul_rn(psi[edge_col(ed)], tri));
          }
        }
      }
      const unsigned s0b = ring_s + 4u * s0n, end_s = ring_s + 4u * RN;
      auto cell_at = [&](unsigned x) {  // shared address of the cell of an edge
        const unsigned c = s0b + x;
        return c >= end_s ? c - 4u * RN : c;
      };
      if (DEL == kSAtomic) {
        // a warp per fired row; two edges per lane per 128-bit load, the
        // loads of up to 256 edges before the first add, and no more than the
        // row has (rows of 11 edges, 3700 a step: 8.5 us a step, 10.0 with all
        // four loads of every row)
        for (int k = warp; k < nf; k += nwarps) {
          const int j = fired[k];
          const int rs = a.row_ptr[j], re = a.row_ptr[j + 1];
          n_events += re - rs;
          for (int e0 = rs & ~1; e0 < re; e0 += 256) {
            uint4 pr[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (e0 + 64 * u >= re) break;
              const int e = e0 + 64 * u + 2 * lane;
              pr[u] = e < re ? *reinterpret_cast<const uint4*>(a.edges + e) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (e0 + 64 * u >= re) break;
              const int e = e0 + 64 * u + 2 * lane;
              const uint2 x = make_uint2(pr[u].x, pr[u].y), y = make_uint2(pr[u].z, pr[u].w);
              auto cell = [&](uint2 ed) {
                const int c = s0n + edge_delay(ed) * nc + edge_col(ed);
                return ring + (c >= RN ? c - RN : c);
              };
              if (e >= rs && e < re) atomicAdd(cell(x), edge_w(x));
              if (e + 1 < re) atomicAdd(cell(y), edge_w(y));
            }
          }
        }
      } else {
        for (int r0 = 0;;) {
          const int nb = min(a.s_cap, nf - r0);
          for (int k0 = 0; k0 < nb && warp < kSRanges; k0 += 32 * kSRows) {
            // lane l: this warp's segments of fired rows k0 + l, k0 + 32 + l, ...
            // Of the batch's events, numbered through the rows: where each
            // segment begins (pos), how many there are, and -- for the first
            // 1024, the usual case all -- a mark at every segment's first
            // event.  Event q of a segment is edge st - pos + q.
            const int nr = min(kSRows, (nb - k0 + 31) >> 5);  // rows of a lane
            int st[kSRows], ln[kSRows], pos[kSRows], total = 0, sg = 0;
            __syncwarp();
            sts_i(mark_s + 4u * lane, 0);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kSRows; ++i) {
              st[i] = ln[i] = pos[i] = 0;
              if (KN && i >= nr) continue;  // warp-uniform; large nets fill them
              if (k0 + 32 * i + lane < nb) {
                const unsigned op = off_w + 4u * ((k0 + 32 * i) * kSOff);
                st[i] = lds_i(op);
                ln[i] = lds_i(op + 4u) - st[i];
              }
              int incl = ln[i];
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
              }
              pos[i] = total + incl - ln[i];
              total += __shfl_sync(0xffffffffu, incl, 31);
              const unsigned ne = __ballot_sync(0xffffffffu, ln[i] > 0);
              if (ln[i] > 0) {
                sts_i(scr_s + 4u * (sg + __popc(ne & below)), st[i] - pos[i]);
                if (pos[i] < 1024) atomicOr(&mark[pos[i] >> 5], 1u << (pos[i] & 31));
              }
              sg += __popc(ne);
            }
            __syncwarp();
            n_events += total;
            unsigned segs = scr_s - 4u;  // last segment begun before the group
            for (int w0 = 0; w0 < total; w0 += 1024) {
              if (w0 > 0) {  // the marks of the next 1024 events
                __syncwarp();
                sts_i(mark_s + 4u * lane, 0);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < kSRows; ++i)
                  if (ln[i] > 0 && (unsigned)(pos[i] - w0) < 1024u)
                    atomicOr(&mark[(pos[i] - w0) >> 5], 1u << ((pos[i] - w0) & 31));
                __syncwarp();
              }
              const int end = min(total, w0 + 1024);
              int ql = w0 + lane;  // this lane's event of the group loaded next
              unsigned mk = mark_s;
              // edges are requested kSAhead groups before they are applied
              uint2 ed[kSAhead];
              auto load = [&](uint2& x) {
                const unsigned M = (unsigned)lds_i(mk);  // (the group behind the last reads a spare word)
                mk += 4u;
                if (ql < end) x = sed[lds_i(segs + 4u * __popc(M & upto)) + ql];
                segs += 4u * __popc(M);
                ql += 32;
              };
#pragma unroll
              for (int u = 0; u < kSAhead; ++u)
                if (w0 + 32 * u < end) load(ed[u]);
              for (int q0 = w0; q0 < end; q0 += 32 * kSAhead) {
#pragma unroll
                for (int u = 0; u < kSAhead; ++u) {
                  const int qu = q0 + 32 * u;
                  if (qu >= end) break;
                  const bool valid = qu + lane < end;
                  const unsigned cell = cell_at(ed[u].x);
                  const float w = __uint_as_float(ed[u].y);
                  if (qu + 32 * kSAhead < end) load(ed[u]);
                  // Every event marks its cell's tag; whoever finds another's
                  // mark there shares its cell with an event of this group.
                  const unsigned tg = tag_s + (((cell - ring_s) >> 2) & tmask);
                  if (valid) sts_b(tg, lane);
                  __syncwarp();
                  int mk = valid ? lds_b(tg) : lane;
                  if (!__any_sync(0xffffffffu, mk != lane)) {
                    if (valid) sts_f(cell, __fadd_rn(lds_f(cell), w));
                    __syncwarp();
                    continue;
                  }
                  // Those of one tag one after another, the earliest first: an
                  // event that finds a later one's mark marks again (the
                  // lowest lane's mark is the one that stays, so this hardly
                  // ever repeats), whoever finds its own mark adds.
                  bool pend = valid;
                  for (;;) {
                    while (__any_sync(0xffffffffu, pend && mk > lane)) {
                      __syncwarp();
                      if (pend && mk > lane) sts_b(tg, lane);
                      __syncwarp();
                      if (pend) mk = lds_b(tg);
                    }
                    if (pend && mk == lane) {
                      sts_f(cell, __fadd_rn(lds_f(cell), w));
                      pend = false;
                    }
                    __syncwarp();
                    if (!__any_sync(0xffffffffu, pend)) break;
                    if (pend) sts_b(tg, lane);
                    __syncwarp();
                    if (pend) mk = lds_b(tg);
                  }
                }
              }
            }
          }
          r0 += a.s_cap;
          if (r0 >= nf) break;
          // more fired rows than s_cap: the next ones' segment starts
          __syncthreads();
          for (int k = warp; k < min(a.s_cap, nf - r0); k += nwarps)
            stage_row(a.sptr, fired[r0 + k] * CL + rank, off + k * kSOff, lane);
          asm volatile("cp.async.wait_all;" ::: "memory");
          __syncthreads();
        }
      }
      __syncthreads();
      s0n = s0n + nc == RN ? 0 : s0n + nc;
    }
    for (int i = tid; i < noc; i += nthr) {
      if (CL == 1) a.counts[(size_t)b * noc + i] = counts[i];
      else if (counts[i]) atomicAdd(&a.counts[(size_t)b * noc + i], counts[i]);
    }
#pragma unroll
    for (int c = 0; c < nch; ++c) {
      const int j = 32 * word_of(c) + lane;
      if (j >= N) continue;
      const float vv = KN ? vr[KN ? c : 0] : sv[j];
      if (a.vfinal) a.vfinal[(size_t)b * N + j] = vv;
      if (a.ro_on && a.ro_rank[j] >= 0) a.ro_v[(size_t)b * a.n_ro + a.ro_rank[j]] = vv;
    }
    const long long te = block_sum_ll(lane == 0 ? n_events : 0, lscratch);
    if (tid == 0) {
      if (CL == 1) a.events[b] = (unsigned long long)te;
      else atomicAdd(&a.events[b], (unsigned long long)te);
      if (rank == 0) a.spikes[b] = (unsigned long long)n_spikes;
    }
    __syncthreads();
  }
  if (CL > 1) cluster_sync();  // no CTA leaves while another may write to it
}

// ---------------------------------------------------------------------------
// tier G / plain: phases of one step for neuron block b of wave slot k
// ---------------------------------------------------------------------------
// Shared memory of a tier-G / plain CTA.  PERSIST (tier G) keeps v / refr
// of its wave slots and cached row / group pointers of its neurons; RSM keeps
// the ring columns of its block ([Bw][R][BS]) for SORT / BUCKET.
struct GSmem {
  float* v;                  // PERSIST [Bw][BS]
  int* refr;                 // PERSIST [Bw][BS]
  int* col;                  // PERSIST [BS]   ring column (global index) or -1
  int* rp;                   // PERSIST [BS+1] row_ptr of the block's neurons
  int* gp;                   // PERSIST [BS+1] gptr of the block's neurons
  int* och;                  // PERSIST [BS]   output channel or -1
  float* ring;               // RSM [Bw][R][BS]
  float* ext;                // [Bw][BS] (one drive buffer per wave slot)
  int* fired;                // [BS]
  int* pa;                   // [P+1]
  int* ib;                   // [P+1] inbox base of every destination block
  int* head;                 // [BS]
  int* tail;                 // [BS]
  unsigned long long* desc;  // [kGDesc]
  unsigned long long* dsort; // [kGDesc]
  int* seg_p;                // [kGDesc]
  int* st_col;               // [kGChunk]
  int* st_slot;              // [kGChunk]
  float* st_w;               // [kGChunk]
  int* st_next;              // [kGChunk]
};

// The arrays a group of threads works in: descriptors, staging, fired list.
__host__ __device__ __forceinline__ size_t g_group_ints(int BS, int P) {
  return 4 * (size_t)kGDesc + kGDesc + 4 * (size_t)kGChunk + ((3 * (size_t)BS + P + 1 + 1) & ~size_t(1));
}

static size_t g_smem_bytes(int BS, int P, int R, int Bw, bool persist, bool rsm, int groups = 1) {
  size_t b = 4 * (g_group_ints(BS, P) * groups + (size_t)Bw * BS + (P + 1));
  if (persist) b += 4 * ((size_t)Bw * BS * 2 + 2 * (size_t)BS + 2 * ((size_t)BS + 1));
  if (rsm) b += 4 * (size_t)Bw * R * BS;
  return b + 64;
}

template <class G>
__device__ __forceinline__ GSmem carve_g(unsigned char* raw, int BS, int P, int R, int Bw,
                                         bool persist, bool rsm, int groups = 1, int group = 0) {
  GSmem s{};
  if constexpr (G::kGroups > 1) raw += 4 * g_group_ints(BS, P) * group;
  s.desc = reinterpret_cast<unsigned long long*>(raw);
  s.dsort = s.desc + kGDesc;
  int* p = reinterpret_cast<int*>(s.dsort + kGDesc);
  if constexpr (G::kGroups == 1) {
    s.ext = reinterpret_cast<float*>(p);
    p += (size_t)Bw * BS;
  }
  s.fired = p;
  s.head = s.fired + BS;
  s.tail = s.head + BS;
  s.pa = s.tail + BS;
  p = s.pa + (P + 1);
  if constexpr (G::kGroups == 1) {
    s.ib = p;
    p += P + 1;
  }
  s.seg_p = p;
  s.st_col = s.seg_p + kGDesc;
  s.st_slot = s.st_col + kGChunk;
  s.st_w = reinterpret_cast<float*>(s.st_slot + kGChunk);
  s.st_next = reinterpret_cast<int*>(s.st_w + kGChunk);
  p = s.st_next + kGChunk;
  if constexpr (G::kGroups > 1) {  // shared by the groups, behind the last
    p = reinterpret_cast<int*>(raw) + g_group_ints(BS, P) * (groups - group);
    s.ext = reinterpret_cast<float*>(p);
    s.ib = p + (size_t)Bw * BS;
    p = s.ib + (P + 1);
  }
  if (persist) {
    s.v = reinterpret_cast<float*>(p);
    s.refr = reinterpret_cast<int*>(s.v + (size_t)Bw * BS);
    s.col = s.refr + (size_t)Bw * BS;
    s.rp = s.col + BS;
    s.gp = s.rp + (BS + 1);
    s.och = s.gp + (BS + 1);
    p = s.och + BS;
  }
  if (rsm) s.ring = reinterpret_cast<float*>(p);
  return s;
}

// Scatter block b's share of step t's injection schedule into ext (dense
// over the block's neurons, zero elsewhere; integration re-zeroes what it
// reads).  Only reads the read-only inputs, so it may run between the arrival
// at and the wait on a grid barrier.
template <class G>
__device__ void load_ext(const G& grp, const FwdArgs& a, float* ext, int sample, long long gstep, int t, int b) {
  __shared__ int s_rng_all[G::kGroups][2];
  int* s_rng = s_rng_all[grp.slot()];
  const int tid = grp.tid(), nthr = grp.size();
  const int lo = b * a.BS, hi = min(a.N, lo + a.BS);
  int k0, k1;
  if (a.sched_blk) {
    const int* sb = a.sched_blk + gstep * (a.P + 1) + b;
    k0 = sb[0];
    k1 = sb[1];
  } else {
    if (tid == 0) {
      const int* sp = a.sched_ptr + a.sptr_off[sample];
      const int q0 = sp[t], q1 = sp[t + 1];
      s_rng[0] = lower_bound_i(a.sched_nid, q0, q1, lo);
      s_rng[1] = lower_bound_i(a.sched_nid, q0, q1, hi);
    }
    grp.sync();
    k0 = s_rng[0];
    k1 = s_rng[1];
    grp.sync();
  }
  for (int q = k0 + tid; q < k1; q += nthr) ext[a.sched_nid[q] - lo] = a.sched_ext[q];
}

// Phase A: drive, integrate / fire the block's neurons, publish the ascending
// fired list, then deliver (ATOMIC) or post inbox descriptors (BUCKET, SORT).
// ext_ready: the drive of this step is already in the slot's ext buffer.
// acc: per-slot spike / event totals in shared memory ([0, kMaxWave) spikes,
// [kMaxWave, 2 kMaxWave) events) that the caller adds to the sample's totals
// once per wave; null: added to the global totals every step.
// EPR: record e-prop's psi and fire counts (the all-SM e-prop forward only).
template <int MODE, bool PERSIST, bool RSM, bool EPR = false, class G = CtaGroup>
__device__ void phase_a(const G& grp, const FwdArgs& a, const GSmem& sm, int* scratch, unsigned long long* acc,
                        int k, int sample, long long gstep, int t, int s0, int b, int cb0, bool ext_ready) {
  const int tid = grp.tid(), nthr = grp.size(), lane = tid & 31, warp = tid >> 5;
  const int nwarps = nthr >> 5;
  const int lo = b * a.BS, hi = min(a.N, lo + a.BS);
  const int R = a.R, nc = a.ncols, N = a.N, BS = a.BS, P = a.P;
  const int par = t & 1;
  float* ext = sm.ext + (PERSIST ? (size_t)k * BS : 0);
  if (!ext_ready) load_ext(grp, a, ext, sample, gstep, t, b);
  grp.sync();
  uint32_t* rast = a.raster ? a.raster + a.raster_off[sample] + (size_t)t * a.W : nullptr;
  int nf = 0;
  long long my_events = 0;
  __shared__ int s_bc_all[G::kGroups][2][32];  // ballot_compact_1 buffers, alternated
  int(*s_bc)[32] = s_bc_all[grp.slot()];
  int bcp = 0;
  for (int base = lo; base < hi; base += nthr) {
    const int j = base + tid, jj = j - lo;
    int f = 0;
    if (j < hi) {
      float vv = PERSIST ? sm.v[k * BS + jj] : a.v[(size_t)k * N + j];
      int rr = PERSIST ? sm.refr[k * BS + jj] : a.refr[(size_t)k * N + j];
      const int c = PERSIST ? sm.col[jj] : a.col_of[j];
      float rin = 0.f;
      if (c >= 0) {
        if (RSM) {
          float* cell = sm.ring + ((size_t)k * R + s0) * BS + (c - cb0);
          rin = *cell;
          *cell = 0.f;
        } else {
          float* cell = a.ring + ((size_t)k * R + s0) * nc + c;
          rin = __ldcg(cell);
          __stcg(cell, 0.f);
        }
      }
      const float e = ext[jj];
      ext[jj] = 0.f;
      float vpre;
      const int oc = PERSIST ? sm.och[jj] : a.out_ch[j];
      f = a.ro_on && oc >= 0 ? readout_step(a.ro_decay, vv, e, rin, EPR ? &vpre : nullptr)
                             : lif_step(a.lif, vv, rr, e, rin, EPR ? &vpre : nullptr);
      if (EPR && c >= 0) {
        // e-prop (cuda_trainer.cu:93-94): the triangular surrogate of this
        // column and step, for the deferred eligibility
        const float thr = a.lif.thr;
        const float dd = __fdiv_rn(fabsf(__fsub_rn(vpre, thr)), thr > 0.f ? thr : 1.f);
        a.psi_hist[((size_t)sample * a.psi_T + t) * nc + c] =
            dd < 1.f ? __fmul_rn(a.gamma, __fsub_rn(1.f, dd)) : 0.f;
      }
      if (PERSIST) {
        sm.v[k * BS + jj] = vv;
        sm.refr[k * BS + jj] = rr;
      } else {
        a.v[(size_t)k * N + j] = vv;
        a.refr[(size_t)k * N + j] = rr;
      }
      if (f) {
        my_events += PERSIST ? sm.rp[jj + 1] - sm.rp[jj] : a.row_ptr[j + 1] - a.row_ptr[j];
        if (MODE != MODE_ATOMIC && PERSIST) {
          // the row's groups are read again when this step's descriptors are
          // posted: start bringing them into L1 while the fired list is built
          const int2* gr = a.groups + sm.gp[jj];
          asm volatile("prefetch.global.L1 [%0];" ::"l"(gr));
          asm volatile("prefetch.global.L1 [%0];" ::"l"(a.groups + max(sm.gp[jj], sm.gp[jj + 1] - 1)));
        }
        if (oc >= 0) atomicAdd(&a.counts[(size_t)sample * a.noc + oc], 1);
        if (EPR && a.fires) atomicAdd(&a.fires[j], 1ull);
      }
    }
    int tot;
    unsigned m;
    const int pos = ballot_compact_1(grp, f, s_bc[bcp], &tot, &m);
    bcp ^= 1;
    if (rast && lane == 0 && base + warp * 32 < hi) rast[(base + warp * 32) >> 5] = m;
    if (f) sm.fired[nf + pos] = j;
    nf += tot;
  }
  grp.sync();
  if (MODE == MODE_SORT) {
    // the ascending fired list, for phase_b_scan (SORT steps whose inbox
    // overflows); the other modes never read it
    int* fo = a.fired + ((size_t)k * 2 + par) * N + lo;
    for (int i = tid; i < nf; i += nthr) __stcg(&fo[i], sm.fired[i]);
  }
  {
    unsigned long long wev = (unsigned long long)my_events;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wev += __shfl_down_sync(0xffffffffu, wev, o);
    if (lane == 0 && wev) atomicAdd(acc ? &acc[kMaxWave + k] : &a.events[sample], wev);
  }
  if (tid == 0) {
    if (MODE == MODE_SORT) __stcg(&a.fired_cnt[((size_t)k * 2 + par) * P + b], nf);
    if (nf) atomicAdd(acc ? &acc[k] : &a.spikes[sample], (unsigned long long)nf);
  }
  if (MODE == MODE_ATOMIC) {
    float* ringk = a.ring + (size_t)k * R * nc;
    for (int q = warp; q < nf; q += nwarps) {
      const int j = sm.fired[q];
      const int rs = PERSIST ? sm.rp[j - lo] : a.row_ptr[j];
      const int re = PERSIST ? sm.rp[j - lo + 1] : a.row_ptr[j + 1];
      for (int e = (rs & ~1) + 2 * lane; e < re; e += 64) {
        const uint4 pr = *reinterpret_cast<const uint4*>(a.gedges + e);
        if (e >= rs) {
          const uint2 ed = make_uint2(pr.x, pr.y);
          atomicAdd(&ringk[(size_t)ring_slot(s0, edge_delay(ed), R) * nc + edge_col(ed)], edge_w(ed));
        }
        if (e + 1 < re) {
          const uint2 ed = make_uint2(pr.z, pr.w);
          atomicAdd(&ringk[(size_t)ring_slot(s0, edge_delay(ed), R) * nc + edge_col(ed)], edge_w(ed));
        }
      }
    }
  } else if (!a.no_post) {
    // one descriptor (first edge, length) per destination block of each
    // fired row; a warp posts the groups of one row in parallel
    int* cnt = a.inbox_cnt + ((size_t)k * 2 + par) * P;
    unsigned long long* box = a.inbox + ((size_t)k * 2 + par) * a.G;
    for (int q = warp; q < nf; q += nwarps) {
      const int j = sm.fired[q];
      const int g0 = PERSIST ? sm.gp[j - lo] : a.gptr[j];
      const int g1 = PERSIST ? sm.gp[j - lo + 1] : a.gptr[j + 1];
      const int re = PERSIST ? sm.rp[j - lo + 1] : a.row_ptr[j + 1];
      for (int g = g0 + lane; g < g1; g += 32) {
        const int2 gr = a.groups[g];
        const int ge = (g + 1 < g1) ? a.groups[g + 1].y : re;
        const int pos = atomicAdd(&cnt[gr.x], 1);
        __stcg(&box[sm.ib[gr.x] + pos],
               ((unsigned long long)(unsigned)gr.y << 32) | (unsigned)(ge - gr.y));
      }
    }
  }
  // no closing barrier: every caller's next step starts with one (the next
  // slot's phase A, grid_arrive, or the end of the launch)
}

// Ring view of one wave slot for the post-owner phase: shared-memory slice
// (local columns, stride BS) or the global ring (global columns, stride ncols).
template <bool RSM>
__device__ __forceinline__ float* ring_base(const FwdArgs& a, const GSmem& sm, int k) {
  return RSM ? sm.ring + (size_t)k * a.R * a.BS : a.ring + (size_t)k * a.R * a.ncols;
}

// SORT fallback when a block's inbox exceeds kGDesc descriptors: walk every
// block's ascending fired list (ascending pre order overall) and stage the
// segments that target this block in that order.
template <bool RSM, class G>
__device__ void phase_b_scan(const G& grp, const FwdArgs& a, const GSmem& sm, int* scratch, int k, int t, int s0,
                             int b, int cb0, int cb1) {
  const int tid = grp.tid(), nthr = grp.size();
  const int R = a.R, P = a.P;
  const int par = t & 1;
  const int* cntk = a.fired_cnt + ((size_t)k * 2 + par) * P;
  const int* fk = a.fired + ((size_t)k * 2 + par) * a.N;
  float* rb = ring_base<RSM>(a, sm, k);
  const int stride = RSM ? a.BS : a.ncols;
  const int col0 = RSM ? 0 : cb0;
  int F;
  {
    const int cnt = tid < P ? __ldcg(&cntk[tid]) : 0;
    const int ex = group_exclusive_scan(grp, cnt, scratch, &F);
    if (tid < P) sm.pa[tid] = ex;
    grp.sync();
  }
  int* seg_s = reinterpret_cast<int*>(sm.desc);
  int* seg_l = reinterpret_cast<int*>(sm.dsort);
  for (int f0 = 0; f0 < F; f0 += nthr) {
    const int f = f0 + tid;
    int gs = 0, gl = 0;
    if (f < F) {
      const int blk = upper_index(sm.pa, P, f);
      const int i = __ldcg(&fk[(size_t)blk * a.BS + (f - sm.pa[blk])]);
      const int g0 = a.gptr[i], g1 = a.gptr[i + 1];
      for (int g = g0; g < g1; ++g) {
        const int2 gr = a.groups[g];
        if (gr.x == b) {
          const int ge = (g + 1 < g1) ? a.groups[g + 1].y : a.row_ptr[i + 1];
          gs = gr.y;
          gl = ge - gr.y;
          break;
        }
        if (gr.x > b) break;
      }
    }
    int nseg;
    unsigned m;
    const int pos = ballot_compact(grp, gl > 0, scratch, &nseg, &m);
    if (gl > 0) {
      seg_s[pos] = gs;
      seg_l[pos] = gl;
    }
    grp.sync();
    int E;
    {
      const int len = tid < nseg ? seg_l[tid] : 0;
      const int ex = group_exclusive_scan(grp, len, scratch, &E);
      if (tid < nseg) sm.seg_p[tid] = ex;
      grp.sync();
    }
    for (int e0 = 0; e0 < E; e0 += kGChunk) {
      const int ce = min(kGChunk, E - e0);
      for (int qq = tid; qq < ce; qq += nthr) {
        const int e = e0 + qq;
        const int s = upper_index(sm.seg_p, nseg, e);
        const uint2 ed = a.gedges[seg_s[s] + (e - sm.seg_p[s])];
        sm.st_slot[qq] = ring_slot(s0, edge_delay(ed), R);
        sm.st_w[qq] = edge_w(ed);
        sm.st_col[qq] = edge_col(ed) - cb0;
      }
      if (ce <= kCountMax)  // apply_cells' table
        for (int i = tid; i < 2 * kCellTable; i += nthr) sm.st_next[i] = 0;
      apply_ordered<!RSM>(grp, ce, sm.head, sm.tail, cb1 - cb0, sm.st_col, sm.st_slot, sm.st_w,
                          sm.st_next, rb, stride, col0);
    }
  }
}

// Phase B for at most 64 inbox descriptors (SORT; 32 for BUCKET) -- the
// common step: warp 0 holds them from the speculative read (lane l:
// descriptors l and l + 32) and scans
// their lengths with shuffles (no rank pass).  BUCKET accumulates straight
// away; SORT stages each event with its gedges index as order key -- within
// one destination block the gedges order is the (pre, edge) order of the CPU
// backend, since gedges keeps the CSR row order and regroups each row stably
// by destination block -- and applies it per ring cell (cell_insert /
// cell_apply with a 1024-key table in the descriptor buffer) with no
// descriptor sort.  Returns false, with nothing applied, for a SORT step of
// more than kFastMax events: the general path takes it.
constexpr int kFastDesc = 64;
constexpr int kFastMax = 512;
constexpr int kFastLen = 16;  // longest segment whose events are written out
static_assert(2 * 2 * kFastMax * sizeof(int) <= kGDesc * sizeof(unsigned long long),
              "the fast path's table lives in the descriptor buffer");

template <int MODE, bool RSM, class G>
__device__ bool phase_b_fast(const G& grp, const FwdArgs& a, const GSmem& sm, int k, int s0, int cb0, int cnt,
                             unsigned long long spec, unsigned long long spec2, bool tail_sync) {
  __shared__ int s_E_all[G::kGroups];
  int& s_E = s_E_all[grp.slot()];
  const int tid = grp.tid(), nthr = grp.size();
  int* tab = reinterpret_cast<int*>(sm.desc);
  if (tid < 32) {
    const unsigned long long d0 = tid < cnt ? spec : 0ull;
    const unsigned long long d1 = MODE == MODE_SORT && tid + 32 < cnt ? spec2 : 0ull;
    const int l0 = (int)(d0 & 0xffffffffu), l1 = (int)(d1 & 0xffffffffu);
    int i0 = l0, i1 = l1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y0 = __shfl_up_sync(0xffffffffu, i0, o), y1 = __shfl_up_sync(0xffffffffu, i1, o);
      if (tid >= o) {
        i0 += y0;
        i1 += y1;
      }
    }
    const int t0 = __shfl_sync(0xffffffffu, i0, 31), all = t0 + __shfl_sync(0xffffffffu, i1, 31);
    // short segments: every event's edge is written out (two or three a
    // descriptor), which saves the threads a search; s_E < 0 says otherwise
    if (all <= kFastMax && !__any_sync(0xffffffffu, l0 > kFastLen || l1 > kFastLen)) {
      const int f0 = (int)(d0 >> 32), f1 = (int)(d1 >> 32);
      for (int i = 0; i < l0; ++i) sm.seg_p[i0 - l0 + i] = f0 + i;
      for (int i = 0; i < l1; ++i) sm.seg_p[t0 + i1 - l1 + i] = f1 + i;
      if (tid == 31) s_E = all;
    } else {
      if (tid < cnt) {
        sm.dsort[tid] = d0;
        sm.seg_p[tid] = i0 - l0;
      }
      if (tid + 32 < cnt) {
        sm.dsort[tid + 32] = d1;
        sm.seg_p[tid + 32] = t0 + i1 - l1;
      }
      if (tid == 31) s_E = ~all;
    }
  }
  if (MODE == MODE_SORT)
    for (int i = tid; i < 2 * 2 * kFastMax; i += nthr) tab[i] = 0;
  grp.sync();
  const bool listed = s_E >= 0;
  const int E = listed ? s_E : ~s_E;
  auto edge_of = [&](int e) {
    if (listed) return sm.seg_p[e];
    const int d = upper_index(sm.seg_p, cnt, e);
    return (int)(sm.dsort[d] >> 32) + (e - sm.seg_p[d]);
  };
  if (MODE == MODE_SORT && (E > kFastMax || E > nthr)) return false;
  const int R = a.R;
  float* rb = ring_base<RSM>(a, sm, k);
  const int stride = RSM ? a.BS : a.ncols;
  const int col0 = RSM ? 0 : cb0;
  if (MODE == MODE_BUCKET) {
    for (int qq = tid; qq < E; qq += nthr) {
      const uint2 ed = a.gedges[edge_of(qq)];
      const int cidx = RSM ? edge_col(ed) - cb0 : edge_col(ed);
      atomicAdd(&rb[(size_t)ring_slot(s0, edge_delay(ed), R) * stride + cidx], edge_w(ed));
    }
    if (tail_sync) grp.sync();
    return true;
  }
  const int q = tid;  // E <= grp.size()
  int c = 0, sl = 0;
  unsigned h = 0;
  bool first = false;
  if (q < E) {
    const int edge = edge_of(q);
    const uint2 ed = a.gedges[edge];
    sl = ring_slot(s0, edge_delay(ed), R);
    c = edge_col(ed) - cb0;
    sm.st_w[q] = edge_w(ed);
    sm.st_slot[q] = edge;  // order key
    h = cell_insert<2 * kFastMax>(tab, sm.st_col, q, c, sl, &first);
  }
  grp.sync();
  if (first)
    cell_apply<!RSM, true, 2 * kFastMax>(tab, sm.st_col, sm.st_slot, sm.st_w, h, q, c, sl, rb, stride,
                                         col0);
  if (tail_sync) grp.sync();
  return true;
}

// Phase B (BUCKET / SORT): as owner of the ring columns of block b, expand
// this step's inbox descriptors and accumulate them into the block's ring
// slice -- unordered (BUCKET) or per ring cell in (pre, edge) order (SORT).
// tail_sync: close with a barrier (another phase B of this step follows;
// otherwise the caller's next step -- phase A, the end of the wave or of the
// launch -- starts with one).
template <int MODE, bool RSM, class G>
__device__ void phase_b(const G& grp, const FwdArgs& a, const GSmem& sm, int* scratch, int k, int t, int s0,
                        int b, int cb0, int cb1, bool tail_sync) {
  __shared__ int s_cnt_all[G::kGroups];
  int& s_cnt = s_cnt_all[grp.slot()];
  if (MODE == MODE_SORT && a.scan_only) {  // partitions: no inbox, every fired list
    phase_b_scan<RSM>(grp, a, sm, scratch, k, t, s0, b, cb0, cb1);
    return;
  }
  const int tid = grp.tid(), nthr = grp.size();
  const int R = a.R;
  const int par = t & 1;
  int* cntp = a.inbox_cnt + ((size_t)k * 2 + par) * a.P + b;
  const unsigned long long* box = a.inbox + ((size_t)k * 2 + par) * a.G + sm.ib[b];
  // read the descriptor slots of the fast path in the same round trip as the
  // count (slots beyond the count hold stale descriptors and are ignored)
  const int cap = sm.ib[b + 1] - sm.ib[b];
  unsigned long long spec = 0, spec2 = 0;
  if (tid < 32 && tid < cap) spec = __ldcg(&box[tid]);
  if (MODE == MODE_SORT && tid < 32 && tid + 32 < cap) spec2 = __ldcg(&box[tid + 32]);
  if (tid == 0) {
    s_cnt = __ldcg(cntp);
    // reset for step t + 2 (written again only after the next grid barrier)
    if (s_cnt) __stcg(cntp, 0);
  }
  grp.sync();
  const int cnt = s_cnt;
  if (cnt == 0) {
    if (tail_sync) grp.sync();  // the next sample's count goes to the same word
    return;
  }
  if (cnt <= (MODE == MODE_SORT ? kFastDesc : 32) &&
      phase_b_fast<MODE, RSM>(grp, a, sm, k, s0, cb0, cnt, spec, spec2, tail_sync))
    return;
  if (MODE == MODE_SORT && cnt > kGDesc) {
    phase_b_scan<RSM>(grp, a, sm, scratch, k, t, s0, b, cb0, cb1);
    return;
  }
  float* rb = ring_base<RSM>(a, sm, k);
  const int stride = RSM ? a.BS : a.ncols;
  const int col0 = RSM ? 0 : cb0;
  for (int d0 = 0; d0 < cnt; d0 += kGDesc) {
    const int dn = min(kGDesc, cnt - d0);
    for (int i = tid; i < dn; i += nthr) sm.desc[i] = __ldcg(&box[d0 + i]);
    grp.sync();
    const unsigned long long* src = sm.desc;
    int E;
    if (dn <= 64) {
      // few descriptors: each finds its rank (by first edge for SORT, by
      // position for BUCKET) and its segment offset in one pass, no scan
      __shared__ int s_E_all[G::kGroups];
      int& s_E = s_E_all[grp.slot()];
      if (tid < dn) {
        const unsigned long long key = sm.desc[tid];
        const unsigned kf = (unsigned)(key >> 32);
        int r = 0, off = 0;
        for (int q = 0; q < dn; ++q) {
          const unsigned long long o = sm.desc[q];
          const bool lt = MODE == MODE_SORT ? (unsigned)(o >> 32) < kf : q < tid;
          r += lt;
          off += lt ? (int)(o & 0xffffffffu) : 0;
        }
        sm.dsort[r] = key;
        sm.seg_p[r] = off;
        if (r == dn - 1) s_E = off + (int)(key & 0xffffffffu);
      }
      grp.sync();
      src = sm.dsort;
      E = s_E;
    } else {
      if (MODE == MODE_SORT) {
        // rank sort by first edge (first edges of distinct rows are distinct)
        for (int i = tid; i < dn; i += nthr) {
          const unsigned long long key = sm.desc[i];
          int r = 0;
          for (int q = 0; q < dn; ++q) r += (sm.desc[q] >> 32) < (key >> 32);
          sm.dsort[r] = key;
        }
        grp.sync();
        src = sm.dsort;
      }
      // prefix of segment lengths, two descriptors per thread at a time
      E = 0;
      for (int q0 = 0; q0 < dn; q0 += 2 * nthr) {
        const int i0 = q0 + 2 * tid, i1 = i0 + 1;
        const int l0 = i0 < dn ? (int)(src[i0] & 0xffffffffu) : 0;
        const int l1 = i1 < dn ? (int)(src[i1] & 0xffffffffu) : 0;
        int part;
        const int ex = E + group_exclusive_scan(grp, l0 + l1, scratch, &part);
        if (i0 < dn) sm.seg_p[i0] = ex;
        if (i1 < dn) sm.seg_p[i1] = ex + l0;
        E += part;
      }
      grp.sync();
    }
    for (int e0 = 0; e0 < E; e0 += kGChunk) {
      const int ce = min(kGChunk, E - e0);
      for (int qq = tid; qq < ce; qq += nthr) {
        const int e = e0 + qq;
        const int d = upper_index(sm.seg_p, dn, e);
        const int edge = (int)(src[d] >> 32) + (e - sm.seg_p[d]);
        const uint2 ed = a.gedges[edge];
        const int slot = ring_slot(s0, edge_delay(ed), R);
        if (MODE == MODE_BUCKET) {
          // shared slice: block-local column; global ring: global column
          const int cidx = RSM ? edge_col(ed) - cb0 : edge_col(ed);
          atomicAdd(&rb[(size_t)slot * stride + cidx], edge_w(ed));
        } else {
          sm.st_slot[qq] = slot;
          sm.st_w[qq] = edge_w(ed);
          sm.st_col[qq] = edge_col(ed) - cb0;
        }
      }
      if (MODE == MODE_SORT) {
        if (ce <= kCountMax)  // apply_cells' table
          for (int i = tid; i < 2 * kCellTable; i += nthr) sm.st_next[i] = 0;
        apply_ordered<!RSM>(grp, ce, sm.head, sm.tail, cb1 - cb0, sm.st_col, sm.st_slot, sm.st_w,
                            sm.st_next, rb, stride, col0);
      } else {
        grp.sync();
      }
    }
  }
}

// Groups (G = WarpGroup): a wave of several samples over small neuron blocks
// leaves most of a CTA idle in every phase of a sample, so a.g_groups groups of
// a.g_threads threads (a thread per neuron of the block, and at least one per
// block for the fired-list scan) take the samples of the wave side by side,
// each group with its own working arrays and a named barrier.  Five uneven
// samples of an 11,931-neuron net (blocks of 96), 232 steps: 3.2 ms one after
// another, 1.5 in four groups.
template <int MODE, bool RSM, bool EPR, class G>
__global__ void __launch_bounds__(kGThreadsMax, 1) k_tier_g(FwdArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int scratch_all[G::kGroups][40];
  __shared__ unsigned long long s_acc[2 * kMaxWave];
  __shared__ int s_samp[kMaxWave], s_T[kMaxWave];
  __shared__ long long s_gb[kMaxWave];
  const int tid = threadIdx.x, nthr = blockDim.x;
  G grp;
  const int ngrp = G::kGroups > 1 ? a.g_groups : 1;
  bool in_group = true;
  if constexpr (G::kGroups > 1) {
    grp.n = a.g_threads;
    grp.g = tid / a.g_threads;
    grp.t = tid - grp.g * a.g_threads;
    in_group = grp.g < ngrp;
  }
  const int gi = G::kGroups > 1 && in_group ? grp.slot() : 0;
  int* scratch = scratch_all[gi];
  const GSmem sm = carve_g<G>(smem_raw, a.BS, a.P, a.R, a.Bw, true, RSM, ngrp, gi);
  const int b = blockIdx.x;
  const int BS = a.BS, R = a.R;
  const int lo = b * BS, hi = min(a.N, lo + BS);
  const int cb0 = a.colbase[b], cb1 = a.colbase[b + 1];
  const unsigned nb = gridDim.x;
  unsigned target = a.stall;
  for (int jj = tid; jj < BS; jj += nthr) {
    sm.col[jj] = lo + jj < hi ? a.col_of[lo + jj] : -1;
    sm.och[jj] = lo + jj < hi ? a.out_ch[lo + jj] : -1;
  }
  if (in_group)
    for (int jj = grp.tid(); jj < BS; jj += grp.size()) {
      sm.head[jj] = -1;
      sm.tail[jj] = -1;
    }
  for (int i = tid; i < a.Bw * BS; i += nthr) sm.ext[i] = 0.f;
  for (int jj = tid; jj <= BS; jj += nthr) {
    const int j = min(lo + jj, hi);
    sm.rp[jj] = a.row_ptr[j];
    sm.gp[jj] = a.gptr[j];
  }
  for (int i = tid; i <= a.P; i += nthr) sm.ib[i] = a.ibase[i];
  const int nwaves = (a.B + a.Bw - 1) / a.Bw;
  for (int w = 0; w < nwaves; ++w) {
    const int q0 = w * a.Bw;
    const int nk = min(a.Bw, a.B - q0);
    if (tid < nk) {
      const int smp = a.order[q0 + tid];
      s_samp[tid] = smp;
      s_T[tid] = a.steps[smp];
      s_gb[tid] = a.stepbase[smp];
      s_acc[tid] = 0;
      s_acc[kMaxWave + tid] = 0;
    }
    for (int i = tid; i < nk * BS; i += nthr) {
      sm.v[i] = 0.f;
      sm.refr[i] = 0;
    }
    if (RSM) {
      for (int i = tid; i < nk * R * BS; i += nthr) sm.ring[i] = 0.f;
    } else {
      const int wcol = cb1 - cb0;
      for (int k = 0; k < nk; ++k) {
        float* ringk = a.ring + (size_t)k * R * a.ncols;
        for (int i = tid; i < R * wcol; i += nthr)
          __stcg(&ringk[(size_t)(i / wcol) * a.ncols + cb0 + (i % wcol)], 0.f);
      }
    }
    target += nb;
    if (!grid_sync(&a.ctl[0], target, a.err, a.wait_ns)) return;
    const int Tw = s_T[0];
    int s0 = 0;  // the step's ring slot
    for (int t = 0; t < Tw; ++t) {
      for (int k = gi; in_group && k < nk; k += ngrp)
        if (t < s_T[k])
          phase_a<MODE, true, RSM, EPR>(grp, a, sm, scratch, s_acc, k, s_samp[k], s_gb[k] + t, t, s0, b, cb0,
                                        t > 0);
      // arrive, fetch the next step's drive while the other blocks catch up,
      // then wait
      target += nb;
      grid_arrive(&a.ctl[0]);
      for (int k = gi; in_group && k < nk; k += ngrp)
        if (t + 1 < s_T[k])
          load_ext(grp, a, sm.ext + (size_t)k * BS, s_samp[k], s_gb[k] + t + 1, t + 1, b);
      if (!grid_wait(&a.ctl[0], target, a.err, a.wait_ns)) return;
      if (MODE != MODE_ATOMIC)
        for (int k = gi; in_group && k < nk; k += ngrp)
          if (t < s_T[k]) {
            bool more = false;
            for (int k2 = k + ngrp; k2 < nk; k2 += ngrp) more |= t < s_T[k2];
            phase_b<MODE, RSM>(grp, a, sm, scratch, k, t, s0, b, cb0, cb1, more);
          }
      s0 = s0 + 1 == R ? 0 : s0 + 1;
    }
    __syncthreads();
    if (tid < nk) {
      if (s_acc[tid]) atomicAdd(&a.spikes[s_samp[tid]], s_acc[tid]);
      if (s_acc[kMaxWave + tid]) atomicAdd(&a.events[s_samp[tid]], s_acc[kMaxWave + tid]);
    }
    if (a.vfinal)
      for (int k = 0; k < nk; ++k)
        for (int j = lo + tid; j < hi; j += nthr)
          a.vfinal[(size_t)s_samp[k] * a.N + j] = sm.v[k * BS + (j - lo)];
    if (a.ro_on)
      for (int k = 0; k < nk; ++k)
        for (int j = lo + tid; j < hi; j += nthr)
          if (sm.och[j - lo] >= 0)
            a.ro_v[(size_t)s_samp[k] * a.n_ro + a.ro_rank[j]] = sm.v[k * BS + (j - lo)];
    target += nb;
    if (!grid_sync(&a.ctl[0], target, a.err, a.wait_ns)) return;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kGThreads) k_plain_a(FwdArgs a, int sample, long long gstep, int t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int scratch[40];
  const GSmem sm = carve_g<CtaGroup>(smem_raw, a.BS, a.P, a.R, 1, false, false);
  for (int jj = threadIdx.x; jj < a.BS; jj += blockDim.x) sm.ext[jj] = 0.f;
  for (int i = threadIdx.x; i <= a.P; i += blockDim.x) sm.ib[i] = a.ibase[i];
  __syncthreads();
  const int b = a.blk0 + blockIdx.x;
  phase_a<MODE, false, false>(CtaGroup(), a, sm, scratch, nullptr, 0, sample, gstep, t, t % a.R, b, a.colbase[b], false);
}

template <int MODE>
__global__ void __launch_bounds__(kGThreads) k_plain_b(FwdArgs a, int t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int scratch[40];
  const GSmem sm = carve_g<CtaGroup>(smem_raw, a.BS, a.P, a.R, 1, false, false);
  for (int jj = threadIdx.x; jj < a.BS; jj += blockDim.x) {
    sm.head[jj] = -1;
    sm.tail[jj] = -1;
  }
  for (int i = threadIdx.x; i <= a.P; i += blockDim.x) sm.ib[i] = a.ibase[i];
  __syncthreads();
  const int b = a.blk0 + blockIdx.x;
  phase_b<MODE, false>(CtaGroup(), a, sm, scratch, 0, t, t % a.R, b, a.colbase[b], a.colbase[b + 1], false);
}

// Zero wave slot 0's global state of block b (plain path, once per sample).
__global__ void k_plain_init(FwdArgs a) {
  const int b = a.blk0 + blockIdx.x;
  const int lo = b * a.BS, hi = min(a.N, lo + a.BS);
  const int cb0 = a.colbase[b], cb1 = a.colbase[b + 1];
  for (int j = lo + threadIdx.x; j < hi; j += blockDim.x) {
    a.v[j] = 0.f;
    a.refr[j] = 0;
  }
  const int w = cb1 - cb0;
  for (int i = threadIdx.x; i < a.R * w; i += blockDim.x)
    a.ring[(size_t)(i / w) * a.ncols + cb0 + (i % w)] = 0.f;
}

__global__ void k_copy_v(FwdArgs a, int sample) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < a.N; j += gridDim.x * blockDim.x) {
    if (a.vfinal) a.vfinal[(size_t)sample * a.N + j] = a.v[j];
    if (a.ro_on && a.ro_rank[j] >= 0) a.ro_v[(size_t)sample * a.n_ro + a.ro_rank[j]] = a.v[j];
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static FwdArgs make_args(Run* r, const snc_lif* lif) {
  const Graph* g = r->g;
  const Inputs* in = r->in;
  FwdArgs a{};
  a.N = g->N; a.S = g->S; a.R = g->R; a.ncols = g->ncols; a.noc = std::max(1, g->noc);
  a.P = g->P; a.BS = g->BS; a.G = g->G;
  a.row_ptr = g->row_ptr; a.edges = g->edges; a.gedges = g->gedges; a.gptr = g->gptr;
  a.groups = g->groups; a.col_of = g->col_of; a.out_ch = g->out_ch; a.colbase = g->colbase;
  a.ibase = g->ibase;
  a.B = in->B; a.order = in->order; a.steps = in->steps; a.sptr_off = in->sptr_off;
  a.stepbase = in->stepbase;
  a.sched_ptr = in->sched_ptr; a.sched_nid = in->sched_nid; a.sched_ext = in->sched_ext;
  a.sched_blk = in->sched_blk;
  a.raster_off = in->raster_off;
  a.counts = r->counts; a.spikes = r->spikes; a.events = r->events;
  a.raster = (r->flags & SNC_B200_RUN_RASTER) ? r->raster : nullptr;
  a.vfinal = (r->flags & SNC_B200_RUN_VFINAL) ? r->vfinal : nullptr;
  a.W = r->W;
  a.Bw = r->Bw; a.v = r->v; a.refr = r->refr; a.ring = r->ring; a.fired = r->fired;
  a.fired_cnt = r->fired_cnt; a.inbox = r->inbox; a.inbox_cnt = r->inbox_cnt;
  a.err = r->err; a.ctl = r->ctl;
  a.lif = LifP{lif->threshold, lif->decay, lif->reset, lif->refractory, lif->reset_mode};
  if (r->edges_w) a.edges = r->edges_w;
  if (r->gedges_w) a.gedges = r->gedges_w;
  a.psi_hist = r->psi_hist;
  a.psi_T = r->psi_T;
  a.fires = r->fires;
  a.gamma = r->gamma;
  a.ro_on = r->ro_decay >= 0.f && r->ro_v && r->ro_logits ? 1 : 0;
  a.ro_decay = a.ro_on ? r->ro_decay : 0.f;
  a.ro_rank = g->ro_rank;
  a.ro_chan = g->ro_chan;
  a.n_ro = g->n_ro;
  a.ro_v = r->ro_v;
  a.ro_logits = r->ro_logits;
  return a;
}

static int ensure_grid_state(Run* r, int Bw) {
  if (r->v && r->Bw_cap >= Bw) {
    r->Bw = Bw;
    return SNC_B200_OK;
  }
  const Graph* g = r->g;
  for (void* p : {(void*)r->v, (void*)r->refr, (void*)r->ring, (void*)r->fired,
                  (void*)r->fired_cnt, (void*)r->inbox, (void*)r->inbox_cnt})
    dev_free(p);
  r->v = nullptr; r->refr = nullptr; r->ring = nullptr; r->fired = nullptr;
  r->fired_cnt = nullptr; r->inbox = nullptr; r->inbox_cnt = nullptr;
  int rc;
  if ((rc = dev_alloc(&r->v, (size_t)Bw * g->N))) return rc;
  if ((rc = dev_alloc(&r->refr, (size_t)Bw * g->N))) return rc;
  if ((rc = dev_alloc(&r->ring, (size_t)Bw * g->R * std::max(1, g->ncols)))) return rc;
  if ((rc = dev_alloc(&r->fired, (size_t)Bw * 2 * g->N))) return rc;
  if ((rc = dev_alloc(&r->fired_cnt, (size_t)Bw * 2 * g->P))) return rc;
  if ((rc = dev_alloc(&r->inbox, (size_t)Bw * 2 * std::max(1, g->G)))) return rc;
  if ((rc = dev_alloc(&r->inbox_cnt, (size_t)Bw * 2 * g->P))) return rc;
  r->Bw = Bw;
  r->Bw_cap = Bw;
  return SNC_B200_OK;
}

static int optin_smem() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin;
}

// Launch shape of the tier-S kernel: neurons of a thread held in registers
// (1 or 2; 0: state in shared memory, beyond 2048 neurons -- four in registers
// took 13.5 us a step for 3000 neurons, 11.5 so), the delivery, fired rows staged at
// once, mask of the conflict tags, bytes of dynamic shared memory.
struct SPlan {
  int kn, del, cap, tmask;
  size_t smem;
};

static SPlan tier_s_layout(const Graph* g, const SLayout& L, int noc, bool inl, int mode, size_t budget) {
  const int nch = std::max(1, (g->N + kSThreads * L.cl - 1) / (kSThreads * L.cl));
  const size_t cells = (size_t)g->R * L.ncols, nw = kSThreads / 32;
  SPlan p{nch <= 1 ? 1 : nch <= 2 ? 2 : 0, kSAtomic, 0, 0, 0};
  auto base = [&](int kn) {
    const size_t cnt = L.cl > 1 ? 2 * ((size_t)g->N + 31) / 32 + 2 : (size_t)(kn ? kn : nch) * nw;
    return (cells + g->N + noc + cnt + (kn ? 0 : 2 * (size_t)g->N) +
            (inl ? (size_t)g->N + g->ncols : 0)) * 4 + (size_t)g->N * 2 + 16;
  };
  p.smem = base(p.kn);
  if (mode != MODE_SORT && L.cl == 1) return p;
  p.del = kSOrdered;
  // a tag per cell before tags per warp (their false conflicts cost more than
  // a second round of staging), then the larger stage; states that leave little
  // room stage few rows at once (one CTA: the last of these always fits beside a
  // state that tier_s_bytes admits).  380 neurons, delays to 149, 240 events a
  // step: 2.2 us a step, 7.3 with a warp's segments one row after another and no
  // scratch, 3.2 with events staged 1024 at a time
  const size_t state = p.smem;
  const struct { int cap, tags; } plans[] = {{g->N > 2048 ? 512 : 256, 0}, {256, 0},  {128, 0},  {256, 512},
                                             {128, 512}, {64, 512}, {64, 256}, {32, 256}, {32, 128}};
  for (const auto& c : plans) {
    if (L.cl > 1 && c.cap < 128) break;
    p.smem = state + nw * s_scratch(c.cap) * 4 + (size_t)c.cap * kSOff * 4 + (c.tags ? nw * c.tags : cells);
    if (p.smem > budget) continue;
    p.cap = c.cap;
    p.tmask = c.tags ? c.tags - 1 : INT_MAX;
    return p;
  }
  return p;  // cap 0: none
}

// A launch of cl CTAs for each of `samples` samples; attr: one attribute, kept
// as long as the configuration.
static cudaLaunchConfig_t s_config(int cl, int samples, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(cl * samples);
  cfg.blockDim = dim3(kSThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = cl;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cl > 1 ? 1 : 0;
  return cfg;
}

template <bool EP>
static int launch_tier_s(const Graph* g, const SLayout& L, int B, int mode, const FwdArgs& a_in, cudaStream_t st) {
  FwdArgs a = a_in;
  using Kern = void (*)(FwdArgs);
  auto pick = [&](int kn, int del, int cap) -> Kern {
    if (L.cl > 1) return k_tier_s<1, EP, kSOrdered, kSCluster>;
    if (del == kSAtomic)
      return kn == 1 ? k_tier_s<1, EP, kSAtomic, 1> : kn == 2 ? k_tier_s<2, EP, kSAtomic, 1>
                                                             : k_tier_s<0, EP, kSAtomic, 1>;
    if (!EP && kn == 1 && cap < 32 * kSRows) return k_tier_s<1, EP, kSRoom, 1>;
    return kn == 1 ? k_tier_s<1, EP, kSOrdered, 1> : kn == 2 ? k_tier_s<2, EP, kSOrdered, 1>
                                                            : k_tier_s<0, EP, kSOrdered, 1>;
  };
  if (L.cl > 1 && EP && a.elig) {
    // its CTAs hold the surrogates of their own columns only
    set_error("tier S: eligibility in the forward needs a whole sample in one CTA");
    return SNC_B200_EUNSUPPORTED;
  }
  cudaFuncAttributes fa{};
  SNCB_CUDA(cudaFuncGetAttributes(&fa, pick(2, kSOrdered, 0)));
  const size_t budget = (size_t)optin_smem() - fa.sharedSizeBytes;
  const SPlan p = tier_s_layout(g, L, a.noc, EP && a.elig, mode, budget);
  if (p.del == kSOrdered && !p.cap) {  // (no such cluster layout is built: tier_s_clusters)
    set_error("tier S: a sample's state does not fit on an SM");
    return SNC_B200_EUNSUPPORTED;
  }
  a.s_cap = p.cap;
  a.s_tmask = p.tmask;
  a.s_nc = L.ncols;
  a.s_col = L.col;
  a.sptr = L.sptr;
  const Kern kern = pick(p.kn, p.del, p.cap);
  SNCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem));
  int per_sm = 0;
  SNCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSThreads, p.smem));
  if (per_sm < 1) {
    set_error("tier S does not fit on an SM");
    return SNC_B200_EUNSUPPORTED;
  }
  cudaLaunchAttribute attr[1];
  const int samples = L.cl > 1 ? B : std::max(1, std::min(B, per_sm * g->sm_count));
  const cudaLaunchConfig_t cfg = s_config(L.cl, samples, p.smem, st, attr);
  SNCB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return SNC_B200_OK;
}

// The layout a batch of B samples runs on: ordered delivery on clusters while
// the device holds all of them at once -- fewer than its SMs would make, since
// a cluster stays within one GPC: 33 of four CTAs on 148 SMs.  34 samples of the
// 1744-neuron net take a second round, 7.2 us a step against 3.8 for 33 and 4.1
// in one CTA each.  (ATOMIC is faster in one CTA, 3.8 against 5.8 us a step at a
// higher rate.)
const SLayout& tier_s_layout_of(const Graph* g, int B, int mode) {
  const SLayout& c = g->sl[1];
  return mode == MODE_SORT && c.sedges && B <= c.max_samples ? c : g->sl[0];
}

// e-prop forward of one minibatch (tier S with eligibility), see eprop.cu.
int launch_eprop_forward(const EpropLaunch& e, cudaStream_t st) {
  const Graph* g = e.g;
  const Inputs* in = e.in;
  if (tier_s_bytes(g->N, g->ncols, g->R, std::max(1, g->noc), e.mode, true, 1024) >
      (size_t)optin_smem()) {
    set_error("e-prop: one sample's state does not fit in one CTA's shared memory");
    return SNC_B200_EUNSUPPORTED;
  }
  FwdArgs a{};
  a.N = g->N; a.S = g->S; a.R = g->R; a.ncols = g->ncols; a.noc = std::max(1, g->noc);
  a.P = g->P; a.BS = g->BS; a.G = g->G;
  a.row_ptr = g->row_ptr; a.edges = e.edges; a.gedges = g->gedges; a.col_of = g->col_of;
  a.out_ch = g->out_ch;
  a.B = in->B; a.order = in->order; a.steps = in->steps; a.sptr_off = in->sptr_off;
  a.stepbase = in->stepbase; a.sched_ptr = in->sched_ptr; a.sched_nid = in->sched_nid;
  a.sched_ext = in->sched_ext; a.raster_off = in->raster_off;
  a.counts = e.counts; a.spikes = e.spikes; a.events = e.events;
  a.W = (g->N + 31) / 32;
  a.err = e.err; a.ctl = e.ctl;
  a.lif = LifP{e.lif.threshold, e.lif.decay, e.lif.reset, e.lif.refractory, e.lif.reset_mode};
  a.elig = e.elig; a.fires = e.fires; a.gamma = e.gamma; a.trace_decay = e.trace_decay;
  a.psi_hist = e.psi_hist; a.psi_T = e.psi_T;
  a.raster = e.raster;
  a.sedges = e.sedges;
  return launch_tier_s<true>(g, *e.layout, in->B, e.mode, a, st);
}

// Wave size and ring placement of the tier-G kernel for this run.
struct GPlan {
  bool rsm;
  int Bw;
  size_t smem;
  int groups, gthreads;  // groups of threads and threads of each (1: the CTA)
};

// want_rsm: -1 automatic (shared-memory ring slices when one sample fits),
// 0 global ring, 1 shared-memory slices (rsm false in the result when they do
// not fit); want_wave: 0 automatic (as many samples as fit), else at most that.
// Static shared memory of the tier-G kernels (the largest instance): the
// dynamic allocation may use what the opt-in limit leaves beside it.
static size_t tier_g_static_smem() {
  static size_t cached = 0;
  static bool done = false;
  if (!done) {
    const void* fns[] = {(const void*)k_tier_g<MODE_ATOMIC, false, false, CtaGroup>,
                         (const void*)k_tier_g<MODE_BUCKET, true, false, CtaGroup>,
                         (const void*)k_tier_g<MODE_BUCKET, false, false, CtaGroup>,
                         (const void*)k_tier_g<MODE_SORT, true, false, CtaGroup>,
                         (const void*)k_tier_g<MODE_SORT, false, false, CtaGroup>,
                         (const void*)k_tier_g<MODE_ATOMIC, false, true, CtaGroup>,
                         (const void*)k_tier_g<MODE_SORT, true, true, CtaGroup>,
                         (const void*)k_tier_g<MODE_SORT, false, true, CtaGroup>};
    size_t m = 0;
    for (const void* f : fns) {
      cudaFuncAttributes fa{};
      if (cudaFuncGetAttributes(&fa, f) == cudaSuccess) m = std::max(m, fa.sharedSizeBytes);
      else cudaGetLastError();
    }
    cached = m;
    done = true;
  }
  return cached;
}

static GPlan plan_tier_g(const Graph* g, int B, int mode, int want_rsm = -1, int want_wave = 0) {
  const size_t optin = (size_t)optin_smem() - std::min((size_t)optin_smem(), tier_g_static_smem());
  GPlan p{false, 1, 0, 1, 0};
  int cap = std::max(1, std::min(B, kMaxWave));
  if (want_wave > 0) cap = std::min(cap, want_wave);
  if (mode != MODE_ATOMIC && want_rsm != 0) {
    int bw = 0;
    while (bw < cap && g_smem_bytes(g->BS, g->P, g->R, bw + 1, true, true) <= optin) ++bw;
    if (bw >= 1) {
      p.rsm = true;
      p.Bw = bw;
    }
  }
  if (!p.rsm) {
    int bw = 0;
    while (bw < cap && g_smem_bytes(g->BS, g->P, g->R, bw + 1, true, false) <= optin) ++bw;
    p.Bw = std::max(1, bw);
  }
  p.smem = g_smem_bytes(g->BS, g->P, g->R, p.Bw, true, p.rsm);
  // groups: a thread per neuron of the block, and per block of the graph; their
  // statics are larger than the single group's by less than this
  constexpr size_t kGroupStatics = 2048;
  p.gthreads = std::max({128, (g->BS + 31) / 32 * 32, (g->P + 31) / 32 * 32});  // (64 descriptors are ranked by a thread each)
  for (int n = std::min({WarpGroup::kGroups, p.Bw, kGThreadsMax / p.gthreads}); n >= 2; --n) {
    const size_t need = g_smem_bytes(g->BS, g->P, g->R, p.Bw, true, p.rsm, n);
    if (need + kGroupStatics > optin) continue;
    p.groups = n;
    p.smem = need;
    // as many threads as a CTA without groups has: two samples of a 1400-neuron
    // net at 500 rows a step, BUCKET, 11.8 us a step, 17.6 with 128 a group
    p.gthreads = std::max(p.gthreads, kGThreads / n / 32 * 32);
    break;
  }
  return p;
}

// Tier-G block size: one thread per neuron of the block when it fits, so the
// integration of a step is a single pass (at least kGThreads, which the
// descriptor prefix scan relies on).
static int tier_g_threads(const Graph* g) {
  return std::max(kGThreads, std::min(kGThreadsMax, (g->BS + 31) / 32 * 32));
}

template <int MODE, bool RSM, bool EPR>
static int launch_tier_g(Run* r, const FwdArgs& a_in, size_t smem, cudaStream_t st) {
  const Graph* g = r->g;
  FwdArgs a = a_in;
  a.g_groups = r->gplan_groups;
  a.g_threads = r->gplan_gthreads;
  int nthr = r->cfg_threads > 0 ? r->cfg_threads : tier_g_threads(g);
  void (*kern)(FwdArgs) = k_tier_g<MODE, RSM, EPR, CtaGroup>;
  if (a.g_groups > 1) {
    kern = k_tier_g<MODE, RSM, EPR, WarpGroup>;
    nthr = std::max(nthr, a.g_groups * a.g_threads);
  }
  SNCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  SNCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nthr, smem));
  if (per_sm * g->sm_count < g->P) {
    set_error("grid tier: blocks cannot be co-resident");
    return SNC_B200_EUNSUPPORTED;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(g->P);
  cfg.blockDim = dim3(nthr);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SNCB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return SNC_B200_OK;
}

template <int MODE>
static int launch_plain(Run* r, FwdArgs a, cudaStream_t st) {
  const Graph* g = r->g;
  const Inputs* in = r->in;
  const int nthr = kGThreads;
  const size_t smem = g_smem_bytes(g->BS, g->P, g->R, 1, false, false);
  SNCB_CUDA(cudaFuncSetAttribute(k_plain_a<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  SNCB_CUDA(cudaFuncSetAttribute(k_plain_b<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int q = 0; q < in->B; ++q) {
    const int smp = in->order_h[q];
    const int T = in->steps_h[smp];
    const long long gb = in->stepbase_h[smp];
    k_plain_init<<<g->P, nthr, 0, st>>>(a);
    for (int t = 0; t < T; ++t) {
      k_plain_a<MODE><<<g->P, nthr, smem, st>>>(a, smp, gb + t, t);
      if (MODE != MODE_ATOMIC) k_plain_b<MODE><<<g->P, nthr, smem, st>>>(a, t);
    }
    if (a.vfinal || a.ro_on)
      k_copy_v<<<std::max(1, std::min(1024, (g->N + 255) / 256)), 256, 0, st>>>(a, smp);
  }
  SNCB_CUDA(cudaGetLastError());
  return SNC_B200_OK;
}

// Some delivery mode runs this graph on tier S (ATOMIC's bound is the least).
bool tier_s_possible(const Graph* g) {
  return tier_s_bytes(g->N, g->ncols, g->R, std::max(1, g->noc), MODE_ATOMIC, false, 1024) <=
         (size_t)optin_smem();
}

// Clusters of layout L that the device holds at once, 0 if a CTA of one lacks the
// room for the ordered delivery.  A part holds the columns of every kSCluster-th
// word of 32 neurons, a quarter of them when they are spread, all of them when
// those words are the ones with synapses.
int tier_s_clusters(const Graph* g, const SLayout& L) {
  int least = 0;
  void (*const kerns[])(FwdArgs) = {k_tier_s<1, false, kSOrdered, kSCluster>, k_tier_s<1, true, kSOrdered, kSCluster>};
  for (auto kern : kerns) {
    cudaFuncAttributes fa{};
    int n = 0;
    bool ok = cudaFuncGetAttributes(&fa, kern) == cudaSuccess;
    const size_t budget = (size_t)optin_smem() - std::min((size_t)optin_smem(), fa.sharedSizeBytes);
    const SPlan p = tier_s_layout(g, L, std::max(1, g->noc), false, MODE_SORT, budget);
    ok = ok && p.cap > 0 &&
         cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget) == cudaSuccess;
    if (ok) {
      cudaLaunchAttribute attr[1];
      const cudaLaunchConfig_t cfg = s_config(L.cl, g->sm_count, p.smem, nullptr, attr);
      ok = cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess;
    }
    cudaGetLastError();
    if (!ok || n < 1) return 0;
    least = least ? std::min(least, n) : n;
  }
  return least;
}

static bool tier_s_fits(const Graph* g, int mode) {
  return tier_s_bytes(g->N, g->ncols, g->R, std::max(1, g->noc), mode, false, 1024) <=
         (size_t)optin_smem();
}

static bool use_tier_s(const Run* r, int mode, int path) {
  return path == SNC_B200_PATH_PERSISTENT && tier_s_fits(r->g, mode) &&
         !(r->flags & SNC_B200_RUN_FORCE_GRID) && r->cfg_tier != 1;
}

int check_shape(const Run* r, int mode, int tier, int threads, int wave, int rsm) {
  const Graph* g = r->g;
  if (tier == 0 && !tier_s_fits(g, mode)) {
    set_error("launch shape: one sample's state does not fit one CTA (tier 0)");
    return SNC_B200_EUNSUPPORTED;
  }
  if (tier < -1 || tier > 1 || wave < 0 || rsm < -1 || rsm > 1 ||
      (threads != 0 && (threads % 32 != 0 || threads < kGThreads || threads > kGThreadsMax))) {
    set_error("launch shape: tier -1..1, threads 0 or a multiple of 32 in [512, 768], wave >= 0, "
              "ring_smem -1..1");
    return SNC_B200_EUNSUPPORTED;
  }
  if (rsm == 1 && mode != MODE_ATOMIC) {
    const GPlan p = plan_tier_g(g, std::max(1, r->in->B), mode, 1, wave);
    if (!p.rsm) {
      set_error("launch shape: ring slices do not fit in shared memory");
      return SNC_B200_EUNSUPPORTED;
    }
  }
  return SNC_B200_OK;
}

static int launch_kernels(Run* r, const FwdArgs& a, int mode, int path, cudaStream_t st);

// Launch body without timing / graph handling: the forward, then the logits
// of the leaky readout units when they are on.
static int launch_body(Run* r, const FwdArgs& a, int mode, int path, cudaStream_t st) {
  int rc = launch_kernels(r, a, mode, path, st);
  if (rc || !a.ro_on) return rc;
  if (r->in->B > 0) {
    k_readout_logits<<<r->in->B, 32, 0, st>>>(a.ro_v, a.ro_chan, a.n_ro, r->in->steps, a.noc,
                                              a.ro_logits);
    SNCB_CUDA(cudaGetLastError());
  }
  return SNC_B200_OK;
}

static int launch_kernels(Run* r, const FwdArgs& a, int mode, int path, cudaStream_t st) {
  if (use_tier_s(r, mode, path)) {
    const SLayout& L = tier_s_layout_of(r->g, r->in->B, mode);
    FwdArgs s = a;
    s.sedges = L.sedges;
    return launch_tier_s<false>(r->g, L, r->in->B, mode, s, st);
  }
  if (path == SNC_B200_PATH_PERSISTENT) {
    const size_t smem = r->gplan_smem;
    if (r->psi_hist || r->fires) {  // e-prop: ATOMIC or SORT delivery
      if (mode == MODE_ATOMIC) return launch_tier_g<MODE_ATOMIC, false, true>(r, a, smem, st);
      if (r->gplan_rsm) return launch_tier_g<MODE_SORT, true, true>(r, a, smem, st);
      return launch_tier_g<MODE_SORT, false, true>(r, a, smem, st);
    }
    if (mode == MODE_ATOMIC) return launch_tier_g<MODE_ATOMIC, false, false>(r, a, smem, st);
    if (r->gplan_rsm) {
      if (mode == MODE_SORT) return launch_tier_g<MODE_SORT, true, false>(r, a, smem, st);
      return launch_tier_g<MODE_BUCKET, true, false>(r, a, smem, st);
    }
    if (mode == MODE_SORT) return launch_tier_g<MODE_SORT, false, false>(r, a, smem, st);
    return launch_tier_g<MODE_BUCKET, false, false>(r, a, smem, st);
  }
  if (mode == MODE_SORT) return launch_plain<MODE_SORT>(r, a, st);
  if (mode == MODE_BUCKET) return launch_plain<MODE_BUCKET>(r, a, st);
  return launch_plain<MODE_ATOMIC>(r, a, st);
}

int launch_run(Run* r, const snc_lif* lif, int mode, int path, cudaStream_t st) {
  const Graph* g = r->g;
  const Inputs* in = r->in;
  if (mode == SNC_B200_MODE_AUTO || path == SNC_B200_PATH_AUTO) {
    int m = mode, p = path, shape[4] = {-1, 0, 0, -1};
    int rc = resolve_auto(g, in, &m, &p, shape);
    if (rc) return rc;
    if (mode == SNC_B200_MODE_AUTO) mode = m;
    if (path == SNC_B200_PATH_AUTO) path = p;
    if (!r->cfg_explicit) {  // the tuned shape, unless the caller set one
      r->cfg_tier = shape[0];
      r->cfg_threads = shape[1];
      r->cfg_wave = shape[2];
      r->cfg_rsm = shape[3];
    }
  }
  if (mode < 0 || mode > MODE_SORT || path < 0 || path > SNC_B200_PATH_PERSISTENT) {
    set_error("bad mode or path");
    return SNC_B200_EINVAL;
  }
  int rc;
  if (!use_tier_s(r, mode, path)) {
    int Bw = 1;
    if (path == SNC_B200_PATH_PERSISTENT) {
      const GPlan p = plan_tier_g(g, in->B, mode, r->cfg_rsm, r->cfg_wave);
      Bw = p.Bw;
      r->gplan_rsm = p.rsm;
      r->gplan_smem = p.smem;
      r->gplan_groups = p.groups;
      r->gplan_gthreads = p.gthreads;
    }
    if ((rc = ensure_grid_state(r, Bw))) return rc;
  }
  FwdArgs a = make_args(r, lif);
  const bool grid = path == SNC_B200_PATH_PERSISTENT && !use_tier_s(r, mode, path);
  const WaitCtl wc = take_wait_ctl(grid && in->B > 0);  // only grid launches wait
  a.wait_ns = wc.ns;
  a.stall = wc.stall;
  const size_t B = (size_t)std::max(1, in->B);
  // The legacy default stream cannot be captured; a run owns a blocking
  // stream (ordered with the legacy stream) that stands in for it.
  if (!st) {
    if (!r->own_stream) SNCB_CUDA(cudaStreamCreate(&r->own_stream));
    st = r->own_stream;
  }
  if (r->outs) {
    SNCB_CUDA(cudaMemsetAsync(r->outs, 0, r->outs_bytes, st));
  } else {
    SNCB_CUDA(cudaMemsetAsync(r->counts, 0, B * std::max(1, g->noc) * sizeof(int), st));
    SNCB_CUDA(cudaMemsetAsync(r->spikes, 0, B * sizeof(unsigned long long), st));
    SNCB_CUDA(cudaMemsetAsync(r->events, 0, B * sizeof(unsigned long long), st));
    SNCB_CUDA(cudaMemsetAsync(r->ctl, 0, 4 * sizeof(unsigned), st));
    SNCB_CUDA(cudaMemsetAsync(r->err, 0, sizeof(int), st));
  }
  if (r->inbox_cnt)
    SNCB_CUDA(cudaMemsetAsync(r->inbox_cnt, 0, (size_t)r->Bw_cap * 2 * g->P * sizeof(int), st));
  if ((r->flags & SNC_B200_RUN_RASTER) && in->raster_words)
    SNCB_CUDA(cudaMemsetAsync(r->raster, 0, (size_t)in->raster_words * sizeof(uint32_t), st));
  SNCB_CUDA(cudaEventRecord(r->ev0, st));
  r->used_graph = false;
  if (in->B > 0) {
    // an injected stall is never captured: the graph keeps the normal launch
    bool use_graph = (r->flags & SNC_B200_RUN_GRAPH) && path == SNC_B200_PATH_PERSISTENT &&
                     !r->graph_refused && a.stall == 0;
    if (use_graph) {
      const int shape[4] = {r->cfg_tier, r->cfg_threads, r->cfg_wave, r->cfg_rsm};
      const bool same = r->gexec && r->gexec_mode == mode && r->gexec_stream == st &&
                        r->gexec_wait_ns == a.wait_ns && r->gexec_ro == (a.ro_on ? a.ro_decay : -1.f) &&
                        std::memcmp(r->gexec_shape, shape, sizeof(shape)) == 0 &&
                        std::memcmp(&r->gexec_lif, lif, sizeof(snc_lif)) == 0;
      if (!same) {
        if (r->gexec) cudaGraphExecDestroy(r->gexec);
        r->gexec = nullptr;
        cudaGraph_t cg = nullptr;
        cudaError_t ce = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
        if (ce == cudaSuccess) {
          rc = launch_body(r, a, mode, path, st);
          ce = cudaStreamEndCapture(st, &cg);
          if (rc) {
            if (cg) cudaGraphDestroy(cg);
            return rc;
          }
          if (ce == cudaSuccess) ce = cudaGraphInstantiate(&r->gexec, cg, 0);
          if (cg) cudaGraphDestroy(cg);
        }
        if (ce != cudaSuccess) {
          // capture refused: remember it and launch directly from now on
          cudaGetLastError();
          r->gexec = nullptr;
          r->graph_refused = true;
          use_graph = false;
        } else {
          r->gexec_mode = mode;
          r->gexec_lif = *lif;
          r->gexec_stream = st;
          r->gexec_wait_ns = a.wait_ns;
          std::memcpy(r->gexec_shape, shape, sizeof(shape));
          r->gexec_ro = a.ro_on ? a.ro_decay : -1.f;
        }
      }
    }
    if (use_graph) {
      SNCB_CUDA(cudaGraphLaunch(r->gexec, st));
      r->used_graph = true;
    } else {
      if ((rc = launch_body(r, a, mode, path, st))) return rc;
    }
  }
  SNCB_CUDA(cudaEventRecord(r->ev1, st));
  r->used_mode = mode;
  r->used_path = path;
  return SNC_B200_OK;
}

// ---------------------------------------------------------------------------
// post-neuron partitions (one sample; the neuron-partitioned C2 mode)
// ---------------------------------------------------------------------------
// Rank r of a partitioned run owns neuron blocks [blk_lo, blk_hi) -- their
// state and ring columns -- and keeps the whole graph.  Per step: integrate
// the own blocks (k_plain_a without inbox posting; spike bits go to the
// raster row of the step), exchange the raster row's words (the caller:
// an all-gather), rebuild every block's ascending fired list from the full
// row (k_mask_fired), then deliver into the own columns by scanning those
// lists in (pre, edge) order (k_plain_b with scan_only): the contributions
// of every ring cell arrive in the serial CPU backend's order, so the union
// of the ranks' results equals a single-device run bit for bit.

// Fired lists and counts of every block from one step's spike bits.
__global__ void k_mask_fired(const uint32_t* __restrict__ mask, int N, int BS, int* fired,
                             int* fired_cnt, int P) {
  __shared__ int scratch[40];
  const int b = blockIdx.x;
  const int lo = b * BS, hi = min(N, lo + BS);
  const int w0 = lo >> 5, w1 = (hi + 31) >> 5;  // BS is a multiple of 32
  int base = 0;
  for (int c0 = w0; c0 < w1; c0 += blockDim.x) {
    const int w = c0 + threadIdx.x;
    uint32_t m = w < w1 ? mask[w] : 0u;
    if (w == w1 - 1 && (hi & 31)) m &= (1u << (hi & 31)) - 1u;  // bits beyond N
    int tot;
    const int ex = block_exclusive_scan(__popc(m), scratch, &tot);
    int pos = base + ex;
    while (m) {
      const int bit = __ffs(m) - 1;
      m &= m - 1u;
      fired[lo + pos++] = (w << 5) + bit;
    }
    base += tot;
  }
  if (threadIdx.x == 0) fired_cnt[b] = base;
}

struct Part {
  Run run;
  int blk_lo = 0, blk_hi = 0;
  snc_lif lif{};
  FwdArgs a{};
  size_t smem = 0;
};

static int part_create(const Graph* g, const Inputs* in, int blk_lo, int blk_hi, const snc_lif* lif,
                       Part* p) {
  if (in->B != 1) { set_error("partition: one sample per run"); return SNC_B200_EINVAL; }
  if (blk_lo < 0 || blk_hi > g->P || blk_lo >= blk_hi) {
    set_error("partition: blocks must satisfy 0 <= block_lo < block_hi <= num_blocks");
    return SNC_B200_EINVAL;
  }
  Run* r = &p->run;
  r->g = g;
  r->in = in;
  r->flags = SNC_B200_RUN_RASTER | SNC_B200_RUN_VFINAL;
  r->W = (g->N + 31) / 32;
  int rc;
  if ((rc = dev_alloc(&r->counts, (size_t)std::max(1, g->noc)))) return rc;
  if ((rc = dev_alloc(&r->spikes, 1))) return rc;
  if ((rc = dev_alloc(&r->events, 1))) return rc;
  if ((rc = dev_alloc(&r->raster, (size_t)std::max<long long>(1, in->raster_words)))) return rc;
  if ((rc = dev_alloc(&r->vfinal, (size_t)std::max(1, g->N)))) return rc;
  if ((rc = dev_alloc(&r->err, 1))) return rc;
  if ((rc = dev_alloc(&r->ctl, 4))) return rc;
  if ((rc = ensure_grid_state(r, 1))) return rc;
  p->blk_lo = blk_lo;
  p->blk_hi = blk_hi;
  p->lif = *lif;
  p->a = make_args(r, lif);
  p->a.blk0 = blk_lo;
  p->a.no_post = 1;
  p->a.scan_only = 1;
  p->smem = g_smem_bytes(g->BS, g->P, g->R, 1, false, false);
  SNCB_CUDA(cudaFuncSetAttribute(k_plain_a<MODE_SORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
  SNCB_CUDA(cudaFuncSetAttribute(k_plain_b<MODE_SORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
  return SNC_B200_OK;
}

static int part_integrate(Part* p, int t, uint32_t* mask, cudaStream_t st) {
  Run* r = &p->run;
  const Graph* g = r->g;
  const int T = r->in->steps_h[0];
  if (t < 0 || t >= T) { set_error("partition: step outside the sample"); return SNC_B200_EINVAL; }
  const int nb = p->blk_hi - p->blk_lo;
  if (t == 0) {
    SNCB_CUDA(cudaMemsetAsync(r->err, 0, sizeof(int), st));
    SNCB_CUDA(cudaMemsetAsync(r->ctl, 0, 4 * sizeof(unsigned), st));
    SNCB_CUDA(cudaMemsetAsync(r->counts, 0, (size_t)std::max(1, g->noc) * sizeof(int), st));
    SNCB_CUDA(cudaMemsetAsync(r->spikes, 0, sizeof(unsigned long long), st));
    SNCB_CUDA(cudaMemsetAsync(r->events, 0, sizeof(unsigned long long), st));
    SNCB_CUDA(cudaMemsetAsync(r->raster, 0, (size_t)std::max<long long>(1, r->in->raster_words) * 4, st));
    k_plain_init<<<nb, kGThreads, 0, st>>>(p->a);
  }
  const long long gb = r->in->stepbase_h[0];
  k_plain_a<MODE_SORT><<<nb, kGThreads, p->smem, st>>>(p->a, 0, gb + t, t);
  SNCB_CUDA(cudaGetLastError());
  if (mask) {  // this partition's words of the step's spike bits
    const size_t w0 = (size_t)p->blk_lo * g->BS / 32;
    const size_t w1 = std::min<size_t>((size_t)r->W, (size_t)p->blk_hi * g->BS / 32);
    if (w1 > w0)
      SNCB_CUDA(cudaMemcpyAsync(mask + w0, r->raster + (size_t)t * r->W + w0, (w1 - w0) * 4,
                                cudaMemcpyDeviceToDevice, st));
  }
  return SNC_B200_OK;
}

static int part_deliver(Part* p, int t, const uint32_t* mask, cudaStream_t st) {
  Run* r = &p->run;
  const Graph* g = r->g;
  const int par = t & 1;
  k_mask_fired<<<g->P, 256, 0, st>>>(mask, g->N, g->BS, r->fired + (size_t)par * g->N,
                                     r->fired_cnt + (size_t)par * g->P, g->P);
  k_plain_b<MODE_SORT><<<p->blk_hi - p->blk_lo, kGThreads, p->smem, st>>>(p->a, t);
  SNCB_CUDA(cudaGetLastError());
  if (t == r->in->steps_h[0] - 1)
    k_copy_v<<<std::max(1, std::min(1024, (g->N + 255) / 256)), 256, 0, st>>>(p->a, 0);
  return SNC_B200_OK;
}

}  // namespace sncb

struct snc_b200_part : sncb::Part {};

using namespace sncb;

extern "C" {

int snc_b200_part_create(const snc_b200_graph* g, const snc_b200_inputs* in, int32_t block_lo,
                         int32_t block_hi, const snc_lif* lif, snc_b200_part** out) {
  if (!g || !in || !lif || !out) { set_error("null argument"); return SNC_B200_EINVAL; }
  *out = nullptr;
  auto* p = new snc_b200_part();
  const int rc = part_create(g, in, block_lo, block_hi, lif, p);
  if (rc) {
    free_run(&p->run);
    delete p;
    return rc;
  }
  *out = p;
  return SNC_B200_OK;
}

int snc_b200_part_release(snc_b200_part* p) {
  if (!p) return SNC_B200_OK;
  free_run(&p->run);
  delete p;
  return SNC_B200_OK;
}

int snc_b200_part_integrate(snc_b200_part* p, int32_t t, uint32_t* mask, void* stream) {
  if (!p) { set_error("null partition"); return SNC_B200_EINVAL; }
  return part_integrate(p, t, mask, static_cast<cudaStream_t>(stream));
}

int snc_b200_part_deliver(snc_b200_part* p, int32_t t, const uint32_t* mask, void* stream) {
  if (!p || !mask) { set_error("null argument"); return SNC_B200_EINVAL; }
  const int T = p->run.in->steps_h[0];
  if (t < 0 || t >= T) { set_error("partition: step outside the sample"); return SNC_B200_EINVAL; }
  return part_deliver(p, t, mask, static_cast<cudaStream_t>(stream));
}

int snc_b200_part_fetch(snc_b200_part* p, float* logits, int64_t* spikes, int64_t* events,
                        uint32_t* raster, float* v_final) {
  if (!p) { set_error("null partition"); return SNC_B200_EINVAL; }
  SNCB_CUDA(cudaDeviceSynchronize());
  int err = 0;
  SNCB_CUDA(cudaMemcpy(&err, p->run.err, 4, cudaMemcpyDeviceToHost));
  if (err) { set_error("device error word set"); return err < 0 ? err : SNC_B200_ECUDA; }
  const Graph* g = p->run.g;
  if (logits && g->noc) {
    std::vector<int> c(g->noc);
    SNCB_CUDA(cudaMemcpy(c.data(), p->run.counts, (size_t)g->noc * 4, cudaMemcpyDeviceToHost));
    for (int k = 0; k < g->noc; ++k) logits[k] = (float)c[k];
  }
  unsigned long long sp = 0, ev = 0;
  SNCB_CUDA(cudaMemcpy(&sp, p->run.spikes, 8, cudaMemcpyDeviceToHost));
  SNCB_CUDA(cudaMemcpy(&ev, p->run.events, 8, cudaMemcpyDeviceToHost));
  if (spikes) *spikes = (int64_t)sp;
  if (events) *events = (int64_t)ev;
  if (raster && p->run.in->raster_words)
    SNCB_CUDA(cudaMemcpy(raster, p->run.raster, (size_t)p->run.in->raster_words * 4, cudaMemcpyDeviceToHost));
  if (v_final) SNCB_CUDA(cudaMemcpy(v_final, p->run.vfinal, (size_t)g->N * 4, cudaMemcpyDeviceToHost));
  return SNC_B200_OK;
}

}  // extern "C"
