// Surrogate-gradient BPTT over the sparse delayed graph: a forward and a
// custom backward kernel behind torch.autograd.Function (snc_b200/bptt.py).
//
// Model (python/snc/model.py:52-72 with the per-synapse delays of
// python/snc/shd_model.py:109-121; restated in oracle/bptt_ref.py):
//   cur_j(t) = sum_{e: post(e)=j} w_e * s_pre(e)(t - d_e)      (0 for t-d < 0)
//   vp_j(t)  = decay * v_j(t-1) + cur_j(t) + ext_j(t)
//   s_j(t)   = H(vp_j(t) - thr)   [smooth variant: x / (1 + k|x|)]
//   v_j(t)   = vp_j(t) * (1 - s_j(t))
// Backward (reverse time), with G = dL/dvp and the fast-sigmoid surrogate
// sg(x) = 1 / (1 + k|x|)^2:
//   gs_i(t)  = dL/ds_i(t) + sum_{e: pre(e)=i} w_e * G_post(e)(t + d_e) - gv_i(t) * vp_i(t)
//   G_i(t)   = gv_i(t) * (1 - s_i(t)) + gs_i(t) * sg(vp_i(t) - thr)
//   gv_i(t-1)= decay * G_i(t);   dL/dext_i(t) = G_i(t)
//   dL/dw_e += G_post(e)(t) * s_pre(e)(t - d_e)
//
// Layout: every per-neuron quantity is [.. ][N][B] with the batch innermost;
// a warp owns a neuron (and a slice of the batch), lanes the samples.  Binary
// spikes are kept as a bit history [T][N][ceil(B/32)].  The incoming edges of a
// neuron are summed in ascending CSR edge order (the order of torch's CPU
// index_add), with separately rounded operations, so the forward spikes equal
// the autograd model's bit for bit.  Steps are separated by a bounded grid
// barrier inside one persistent cooperative launch.  With checkpointing (every
// K steps) only v at segment ends is stored; the backward recomputes vp for
// one segment at a time from those checkpoints and the stored spikes.
//
// k_res_forward / k_res_backward run binary spikes when every warp's edges fit
// shared memory and all warps are co-resident (up to 32 an SM, degrees up to
// 256); k_bptt_forward / k_bptt_backward take everything else (the smoothed
// variant, larger graphs) and give the same bits.  Measured: 4096 recurrent
// neurons, fan-in 64, 64 samples, 256 steps: forward 1.02 ms, backward 3.21 ms
// (1.9 and 6.8 with the general form, a warp per neuron walking all spike words
// and gradients through shuffles, its weight gradients before the barrier);
// 784-512-512 at 128 samples, 100 steps: 0.59 and 1.68 ms (1.0 and 3.57).
// What is left is latency: a grid barrier and two L2 trips a step, and in the
// backward 458 KB of gradients an SM gathers from L2 each step (7000 cycles at
// 64 B a cycle, of 27000).
#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

struct snc_b200_bptt {
  int N = 0, S = 0, D = 1, R = 2, sm_count = 0;
  int max_deg = 0;     // largest in- or out-degree
  bool even = false;   // runs of 32 neurons have about the same number of edges
  int resident = 1;    // allow resident launches
  int *row_ptr = nullptr, *out_post = nullptr, *out_d = nullptr;
  int *col_ptr = nullptr, *in_pre = nullptr, *in_d = nullptr, *in_eidx = nullptr;
  float *v = nullptr, *gv = nullptr, *gcur = nullptr, *seg = nullptr, *part = nullptr;
  size_t v_cap = 0, gv_cap = 0, gcur_cap = 0, seg_cap = 0, part_cap = 0;
  unsigned* ctl = nullptr;
  int* err = nullptr;
};

namespace sncb {

struct BpArgs {
  int N, S, R, T, B, K, smooth;
  float thr, decay, slope;
  const int *row_ptr, *out_post, *out_d, *col_ptr, *in_pre, *in_d, *in_eidx;
  const float* w;
  const float* ext;    // [T][N][B]
  float* spikes;       // [T][N][B]
  uint32_t* bits;      // [T][N][KB]
  float* vsaved;       // K > 0: [T/K][N][B] v at segment ends; K == 0: [T][N][B] vp
  float* v;            // [N][B]
  const float* gspk;   // [T][N][B]
  float* gext;         // [T][N][B] or null
  float* gv;           // [N][B]
  float* gcur;         // [R][N][B]
  float* seg;          // [K][N][B]
  unsigned* ctl;
  int* err;
  int KBs;             // 32-sample words of a bit row: ceil(B / 32)
  int SL, VB, VB_log;  // batch slices of the weight gradient, words of a slice (1, 2 or 4)
  int split;           // the sums are those of the resident launches
  float* part;         // [SL][S] weight gradient of every slice (one: the weight gradient)
  int Bp;              // resident backward: floats of a row (B, rounded up to 8, a smaller batch to VB)
  float* ring;         // resident backward: [R][N][Bp] future gradients
  int res_cap;         // resident launches: edges per direction staged per warp
  int even;            // resident launches: items in order, not round the CTAs
  unsigned long long wait_ns;  // grid-barrier wait bound (0: the default)
  unsigned stall;              // injected arrivals that never come (failure tests)
};

constexpr int kBpThreads = 256;
// Blocks per SM the kernels are compiled for: one warp per neuron has to stay
// co-resident (4096 neurons need 4 blocks of 8 warps on each of 148 SMs), so
// narrow batches keep to 64 registers.
template <int KB>
constexpr int kBpMinBlocks = KB <= 2 ? 4 : (KB <= 4 ? 2 : 1);
constexpr int kResCapMax = 256;  // largest in / out degree a resident launch stages

// A resident launch gives every warp one neuron for the whole launch and
// stages that neuron's edges in shared memory once: incoming (pre, delay,
// weight, CSR edge index, weight-gradient accumulator) in ascending CSR edge
// order, outgoing (post, delay, weight) in CSR order.  The per-step edge
// metadata loads and the global weight-gradient read-modify-writes leave the
// time loop; the arithmetic and its order are those of the global-memory form.
struct WarpEdges {
  int *in_pre, *in_d, *in_eidx;
  float *in_w, *in_acc;
  int *out_post, *out_d;
  float* out_w;
  int nin, nout;
};

// Shared memory of a resident launch per warp: 8 arrays of res_cap entries.
__device__ __forceinline__ WarpEdges warp_edges(float* base, int cap) {
  const int wib = threadIdx.x >> 5;
  int* p = reinterpret_cast<int*>(base) + (size_t)wib * 8 * cap;
  WarpEdges we;
  we.in_pre = p;
  we.in_d = p + cap;
  we.in_eidx = p + 2 * cap;
  we.in_w = reinterpret_cast<float*>(p + 3 * cap);
  we.in_acc = reinterpret_cast<float*>(p + 4 * cap);
  we.out_post = p + 5 * cap;
  we.out_d = p + 6 * cap;
  we.out_w = reinterpret_cast<float*>(p + 7 * cap);
  we.nin = we.nout = 0;
  return we;
}

// Stage neuron i's edges (the whole warp; i < N).
__device__ __forceinline__ void stage_edges(const BpArgs& a, int i, WarpEdges& we) {
  const int lane = threadIdx.x & 31;
  const int c0 = a.col_ptr[i], r0 = a.row_ptr[i];
  we.nin = a.col_ptr[i + 1] - c0;
  we.nout = a.row_ptr[i + 1] - r0;
  for (int e = lane; e < we.nin; e += 32) {
    we.in_pre[e] = a.in_pre[c0 + e];
    we.in_d[e] = a.in_d[c0 + e];
    const int ei = a.in_eidx[c0 + e];
    we.in_eidx[e] = ei;
    we.in_w[e] = a.w[ei];
    we.in_acc[e] = 0.f;
  }
  for (int e = lane; e < we.nout; e += 32) {
    we.out_post[e] = a.out_post[r0 + e];
    we.out_d[e] = a.out_d[r0 + e];
    we.out_w[e] = a.w[r0 + e];
  }
  __syncwarp();
}

// One step of the forward for neuron j.  v holds the neuron's state before
// the step (per lane, batch elements lane + 32k) and is updated; vp receives
// the pre-reset potential; s the spike.
// Edges whose spike words / future gradients one lane keeps in flight.
template <int KB>
constexpr int kEdgeBatch = KB >= 8 ? 4 : 8;

template <int KB, bool SMOOTH, bool RES>
__device__ __forceinline__ void fwd_neuron(const BpArgs& a, int t, int j, float (&v)[KB],
                                           float (&vp)[KB], float (&s)[KB], const WarpEdges& we) {
  const int lane = threadIdx.x & 31;
  float acc[KB];
#pragma unroll
  for (int k = 0; k < KB; ++k) acc[k] = 0.f;
  const int e0 = RES ? 0 : a.col_ptr[j], e1 = RES ? we.nin : a.col_ptr[j + 1];
  // one lane per incoming edge of a 32-edge group: its pre, delay, weight
  // and (step form) the spike words of its pre at t - d
  auto group = [&](int eb, int& pre, int& d, float& w, uint32_t (&mw)[KB]) {
    const int n = min(32, e1 - eb);
    pre = 0;
    d = 1 << 30;
    w = 0.f;
    if (lane < n) {
      pre = RES ? we.in_pre[eb + lane] : a.in_pre[eb + lane];
      d = RES ? we.in_d[eb + lane] : a.in_d[eb + lane];
      w = RES ? we.in_w[eb + lane] : a.w[a.in_eidx[eb + lane]];
    }
    if constexpr (!SMOOTH) {
      const bool ok = lane < n && t - d >= 0;
      const uint32_t* wp = a.bits + ((size_t)(ok ? t - d : 0) * a.N + pre) * a.KBs;
#pragma unroll
      for (int k = 0; k < KB; ++k) mw[k] = ok && k < a.KBs ? wp[k] : 0u;
    }
  };
  int my_pre, my_d;
  float my_w;
  uint32_t mw[KB];
  if (e0 < e1) group(e0, my_pre, my_d, my_w, mw);
  for (int eb = e0; eb < e1; eb += 32) {
    const int n = min(32, e1 - eb);
    if constexpr (!SMOOTH) {
      // the next group's spike words are requested before this group's are
      // added: the words of 64 edges are one round trip; the words are
      // broadcast by shuffles and added in edge order (the order of the sum
      // is unchanged)
      int nx_pre = 0, nx_d = 0;
      float nx_w = 0.f;
      uint32_t nx_mw[KB];
      if (eb + 32 < e1) group(eb + 32, nx_pre, nx_d, nx_w, nx_mw);
      for (int q = 0; q < n; ++q) {
        const float ww = __shfl_sync(0xffffffffu, my_w, q);
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const uint32_t word = __shfl_sync(0xffffffffu, mw[k], q);
          if ((word >> lane) & 1u) acc[k] = __fadd_rn(acc[k], ww);
        }
      }
      my_pre = nx_pre;
      my_d = nx_d;
      my_w = nx_w;
#pragma unroll
      for (int k = 0; k < KB; ++k) mw[k] = nx_mw[k];
    } else {
      for (int q = 0; q < n; ++q) {
        const int pre = __shfl_sync(0xffffffffu, my_pre, q);
        const int d = __shfl_sync(0xffffffffu, my_d, q);
        const float ww = __shfl_sync(0xffffffffu, my_w, q);
        const int ts = t - d;
        if (ts < 0) continue;
        const float* sp = a.spikes + ((size_t)ts * a.N + pre) * a.B;
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const int b = 32 * k + lane;
          if (b < a.B) acc[k] = __fadd_rn(acc[k], __fmul_rn(ww, sp[b]));
        }
      }
      if (eb + 32 < e1) group(eb + 32, my_pre, my_d, my_w, mw);
    }
  }
#pragma unroll
  for (int k = 0; k < KB; ++k) {
    const int b = 32 * k + lane;
    const float x_ext = b < a.B ? a.ext[((size_t)t * a.N + j) * a.B + b] : 0.f;
    vp[k] = __fadd_rn(__fadd_rn(__fmul_rn(a.decay, v[k]), acc[k]), x_ext);
    const float x = __fsub_rn(vp[k], a.thr);
    s[k] = SMOOTH ? __fdiv_rn(x, __fadd_rn(1.f, __fmul_rn(a.slope, fabsf(x)))) : (x >= 0.f ? 1.f : 0.f);
    v[k] = __fmul_rn(vp[k], __fsub_rn(1.f, s[k]));
  }
}

template <int KB, bool SMOOTH, bool RES>
__global__ void __launch_bounds__(kBpThreads, kBpMinBlocks<KB>) k_bptt_forward(BpArgs a) {
  extern __shared__ float sm_all[];
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int W = (gridDim.x * blockDim.x) >> 5;
  const unsigned nb = gridDim.x;
  unsigned target = a.stall;
  WarpEdges we{};
  if (RES) {
    we = warp_edges(sm_all, a.res_cap);
    if (gw < a.N) stage_edges(a, gw, we);
  }
  for (int j = gw; j < a.N; j += W)
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      const int b = 32 * k + lane;
      if (b < a.B) a.v[(size_t)j * a.B + b] = 0.f;
    }
  for (int t = 0; t < a.T; ++t) {
    for (int j = gw; j < a.N; j += W) {
      float v[KB], vp[KB], s[KB];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int b = 32 * k + lane;
        v[k] = b < a.B ? a.v[(size_t)j * a.B + b] : 0.f;
      }
      fwd_neuron<KB, SMOOTH, RES>(a, t, j, v, vp, s, we);
      const size_t plane = ((size_t)t * a.N + j) * a.B;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int b = 32 * k + lane;
        const bool ok = b < a.B;
        if (ok) {
          a.v[(size_t)j * a.B + b] = v[k];
          a.spikes[plane + b] = s[k];
          if (a.K == 0) a.vsaved[plane + b] = vp[k];
          else if ((t + 1) % a.K == 0 || t + 1 == a.T) a.vsaved[((size_t)(t / a.K) * a.N + j) * a.B + b] = v[k];
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok && s[k] != 0.f);
        if (!SMOOTH && lane == 0 && k < a.KBs) a.bits[((size_t)t * a.N + j) * a.KBs + k] = m;
      }
    }
    target += nb;
    if (!grid_sync(&a.ctl[0], target, a.err, a.wait_ns)) return;
  }
}

// One backward step for neuron i; vp_plane points at the [N][B] plane of
// pre-reset potentials of step t.  sm_g: this warp's [B] scratch.
template <int KB, bool SMOOTH, bool RES, bool SPLIT>
__device__ __forceinline__ void bwd_neuron(const BpArgs& a, int t, int i, const float* vp_plane,
                                           float* sm_g, const WarpEdges& we) {
  const int lane = threadIdx.x & 31;
  const int N = a.N, B = a.B;
  // SPLIT: two sums, each in edge order: the upstream gradient with the synapses
  // of delay 2 and more, and those of delay 1 (k_res_backward takes the first
  // before the barrier of the step); else one
  float gs[KB], g1[KB];
  const size_t plane = ((size_t)t * N + i) * B;
#pragma unroll
  for (int k = 0; k < KB; ++k) {
    const int b = 32 * k + lane;
    gs[k] = b < B ? a.gspk[plane + b] : 0.f;
    g1[k] = 0.f;
  }
  // gradient reaching s_i(t) through every outgoing synapse (fires at t + d)
  const int tr = t % a.R;
  const int e0 = RES ? 0 : a.row_ptr[i], e1 = RES ? we.nout : a.row_ptr[i + 1];
  for (int eb = e0; eb < e1; eb += 32) {
    const int n = min(32, e1 - eb);
    int my_post = 0, my_d = 1 << 30;
    float my_w = 0.f;
    if (lane < n) {
      my_post = RES ? we.out_post[eb + lane] : a.out_post[eb + lane];
      my_d = RES ? we.out_d[eb + lane] : a.out_d[eb + lane];
      my_w = RES ? we.out_w[eb + lane] : a.w[eb + lane];
    }
    // each lane turns its own edge into an offset into the ring of future
    // gradients (slot of t + d: one conditional subtraction, d < R) and a
    // validity bit; the batches below only broadcast them
    const unsigned okm = __ballot_sync(0xffffffffu, lane < n && t + my_d < a.T);
    const unsigned onem = SPLIT ? __ballot_sync(0xffffffffu, lane < n && my_d == 1) : 0u;
    size_t my_off = 0;
    if ((okm >> lane) & 1u) {
      const int slot = tr + my_d >= a.R ? tr + my_d - a.R : tr + my_d;
      my_off = ((size_t)slot * N + my_post) * B;
    }
    // the future gradients of kEdgeBatch edges are loaded together, then
    // accumulated in edge order
    for (int q0 = 0; q0 < n; q0 += kEdgeBatch<KB>) {
      float gv[kEdgeBatch<KB>][KB];
      float wwv[kEdgeBatch<KB>];
      bool okv[kEdgeBatch<KB>];
#pragma unroll
      for (int u = 0; u < kEdgeBatch<KB>; ++u) {
        const int src = (q0 + u) & 31;  // q0 + u < 32: kEdgeBatch divides 32
        const unsigned olo = __shfl_sync(0xffffffffu, (unsigned)my_off, src);
        const unsigned ohi = __shfl_sync(0xffffffffu, (unsigned)(my_off >> 32), src);
        wwv[u] = __shfl_sync(0xffffffffu, my_w, src);
        okv[u] = (okm >> src) & 1u;
        const float* gp = a.gcur + (((size_t)ohi << 32) | olo);
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const int b = 32 * k + lane;
          gv[u][k] = okv[u] && b < B ? gp[b] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < kEdgeBatch<KB>; ++u)
        if (okv[u])
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            const int b = 32 * k + lane;
            if (b >= B) continue;
            if (SPLIT && (onem >> ((q0 + u) & 31)) & 1u) g1[k] = __fmaf_rn(wwv[u], gv[u][k], g1[k]);
            else gs[k] = __fmaf_rn(wwv[u], gv[u][k], gs[k]);
          }
    }
  }
  float* gc = a.gcur + ((size_t)tr * N + i) * B;
#pragma unroll
  for (int k = 0; k < KB; ++k) {
    const int b = 32 * k + lane;
    if (b >= B) continue;
    const float vp = vp_plane[(size_t)i * B + b];
    const float x = __fsub_rn(vp, a.thr);
    const float den = __fadd_rn(1.f, __fmul_rn(a.slope, fabsf(x)));
    const float s = SMOOTH ? __fdiv_rn(x, den) : (x >= 0.f ? 1.f : 0.f);
    const float sg = __fdiv_rn(1.f, __fmul_rn(den, den));
    const float gvv = a.gv[(size_t)i * B + b];
    const float gst = __fsub_rn(SPLIT ? __fadd_rn(gs[k], g1[k]) : gs[k], __fmul_rn(gvv, vp));
    const float g = __fadd_rn(__fmul_rn(gvv, __fsub_rn(1.f, s)), __fmul_rn(gst, sg));
    gc[b] = g;
    if (a.gext) a.gext[plane + b] = g;
    a.gv[(size_t)i * B + b] = __fmul_rn(a.decay, g);
    sm_g[b] = g;
  }
  __syncwarp();
  // dL/dw for every incoming synapse: lane per synapse, sum of G over the
  // samples whose pre neuron fired at t - d (only set bits are visited);
  // the spike words of a lane's next two synapses are loaded together
  const int c0 = RES ? 0 : a.col_ptr[i], c1 = RES ? we.nin : a.col_ptr[i + 1];
  for (int e = c0 + lane; e < c1; e += 64) {
    int ts[2], pre[2];
    uint32_t wv[2][KB];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int eu = e + 32 * u;
      ts[u] = -1;
      pre[u] = 0;
      if (eu < c1) {
        ts[u] = t - (RES ? we.in_d[eu] : a.in_d[eu]);
        pre[u] = RES ? we.in_pre[eu] : a.in_pre[eu];
      }
      if (!SMOOTH) {
        const uint32_t* wp = a.bits + ((size_t)(ts[u] >= 0 ? ts[u] : 0) * N + pre[u]) * a.KBs;
#pragma unroll
        for (int k = 0; k < KB; ++k) wv[u][k] = ts[u] >= 0 && k < a.KBs ? wp[k] : 0u;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (ts[u] < 0) continue;
      const int eu = e + 32 * u;
      float c = 0.f;
      auto add = [&](size_t slice) {  // to the weight gradient of one batch slice
        if (c == 0.f) return;
        if (RES) {
          we.in_acc[eu] = __fadd_rn(we.in_acc[eu], c);
        } else {
          float* gp = a.part + slice * a.S + a.in_eidx[eu];
          *gp = __fadd_rn(*gp, c);
        }
      };
      if (!SMOOTH) {
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          uint32_t word = wv[u][k];
          while (word) {
            const int bb = __ffs(word) - 1;
            c = __fadd_rn(c, sm_g[32 * k + bb]);
            word &= word - 1u;
          }
          // SPLIT: a sum per slice of VB words (KB is a multiple of VB)
          if (SPLIT && ((k + 1) & (a.VB - 1)) == 0) {
            add((size_t)(k >> a.VB_log));
            c = 0.f;
          }
        }
      } else {
        const float* sp = a.spikes + ((size_t)ts[u] * N + pre[u]) * B;
        for (int b = 0; b < B; ++b) c = __fadd_rn(c, __fmul_rn(sm_g[b], sp[b]));
      }
      if (!SPLIT) add(0);
    }
  }
  __syncwarp();
}

// Staged edges: the warp's weight gradients, accumulated in shared memory in the
// order the global form adds them, go out once.
__device__ __forceinline__ void flush_acc(const BpArgs& a, const WarpEdges& we) {
  const int lane = threadIdx.x & 31;
  for (int e = lane; e < we.nin; e += 32) a.part[we.in_eidx[e]] = we.in_acc[e];
}

// The weight gradient: the slices' sums in slice order.
__global__ void k_sum_slices(int S, int SL, const float* __restrict__ part, float* __restrict__ gw) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < S; e += gridDim.x * blockDim.x) {
    float x = part[e];
    for (int sl = 1; sl < SL; ++sl) x = __fadd_rn(x, part[(size_t)sl * S + e]);
    gw[e] = x;
  }
}

template <int KB, bool SMOOTH, bool RES, bool SPLIT>
__global__ void __launch_bounds__(kBpThreads, kBpMinBlocks<KB>) k_bptt_backward(BpArgs a) {
  extern __shared__ float sm_all[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  float* sm_g = sm_all + (size_t)wib * (32 * KB);
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int W = (gridDim.x * blockDim.x) >> 5;
  const unsigned nb = gridDim.x;
  const size_t NB = (size_t)a.N * a.B;
  unsigned target = a.stall;
  WarpEdges we{};
  if (RES) {
    we = warp_edges(sm_all + (size_t)(blockDim.x >> 5) * 32 * KB, a.res_cap);
    if (gw < a.N) stage_edges(a, gw, we);
  }
  for (int i = gw; i < a.N; i += W)
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      const int b = 32 * k + lane;
      if (b < a.B) a.gv[(size_t)i * a.B + b] = 0.f;
    }
  if (a.K == 0) {
    for (int t = a.T - 1; t >= 0; --t) {
      for (int i = gw; i < a.N; i += W)
        bwd_neuron<KB, SMOOTH, RES, SPLIT>(a, t, i, a.vsaved + (size_t)t * NB, sm_g, we);
      target += nb;
      if (!grid_sync(&a.ctl[0], target, a.err, a.wait_ns)) return;
    }
    if (RES) flush_acc(a, we);
    return;
  }
  const int nseg = (a.T + a.K - 1) / a.K;
  for (int sg = nseg - 1; sg >= 0; --sg) {
    const int t0 = sg * a.K, t1 = min(a.T, t0 + a.K);
    // recompute the segment's pre-reset potentials of this warp's neurons
    // from the checkpoint and the stored spikes (no cross-neuron dependence)
    for (int i = gw; i < a.N; i += W) {
      float v[KB], vp[KB], s[KB];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int b = 32 * k + lane;
        v[k] = (sg > 0 && b < a.B) ? a.vsaved[(size_t)(sg - 1) * NB + (size_t)i * a.B + b] : 0.f;
      }
      for (int t = t0; t < t1; ++t) {
        fwd_neuron<KB, SMOOTH, RES>(a, t, i, v, vp, s, we);
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const int b = 32 * k + lane;
          if (b < a.B) a.seg[(size_t)(t - t0) * NB + (size_t)i * a.B + b] = vp[k];
        }
      }
    }
    for (int t = t1 - 1; t >= t0; --t) {
      for (int i = gw; i < a.N; i += W)
        bwd_neuron<KB, SMOOTH, RES, SPLIT>(a, t, i, a.seg + (size_t)(t - t0) * NB, sm_g, we);
      target += nb;
      if (!grid_sync(&a.ctl[0], target, a.err, a.wait_ns)) return;
    }
  }
  if (RES) flush_acc(a, we);
}

// ---------------------------------------------------------------------------
// Resident binary-spike launches: one warp per (neuron, batch slice of VB
// 32-sample words), all co-resident, one CTA per SM.
// ---------------------------------------------------------------------------
// Forward.  The spike words of 32 in-edges (lane: edge) are turned into one
// word per sample (a 32 x 32 bit transpose by shuffles); every sample then adds
// the weights of its set bits in edge order, a bit test and a predicated add
// per edge (following the set bits alone saves instructions but waits for a
// shared-memory load per spike).  Words of delay 2 and more are requested
// before the step's barrier, spikes and drive move behind the arrival.
//
// Backward.  G of a step depends on the previous step's only through the
// synapses of delay 1.  Everything else -- the gather over the other synapses,
// the weight gradient, the recomputation of a checkpoint segment -- runs
// between the arrival at a step's barrier and the wait for it.  G lies in a
// ring whose rows start on VB floats, read as VB-wide vectors; lanes beyond the
// batch read the next row (there is room behind the last) and drop what they
// get.  Rows of steps beyond T are zero.  Edge offsets of a step are computed
// once per edge and passed through shared memory.  The last steps, as many as
// the largest delay, stage the edges anew with weight 0 for those that reach
// beyond T (an infinite weight times a zero gradient would be NaN), about 2 us a
// step, so the gather needs no check (one per offset took 1.7 % of the backward
// of 4096 neurons, 256 steps).
//
// Items go round the CTAs (item i to CTA i mod grid), so that neurons without
// synapses in one direction share an SM with others; where every run of 32
// neurons has about the same number of edges (a.even) they are dealt in
// order, and neighbours of a net with local synapses find rows that they share
// in L1.  4096 neurons on a ring, 64 samples: backward 3487 -> 3240 us,
// forward 1057 -> 1023; the layers of 784, 512 and 512 neurons in order would
// take 1869 and 740 us instead of 1705 and 594.

template <int VB>
struct VecOf;
template <>
struct VecOf<1> { typedef float T; };
template <>
struct VecOf<2> { typedef float2 T; };
template <>
struct VecOf<4> { typedef float4 T; };

// 32-edge groups whose words are requested at once
template <int VB>
constexpr int kRsGroups = VB == 1 ? 8 : VB == 2 ? 5 : 3;

// Shared memory of one warp, in ints: in-edges (base of the pre's words,
// delay, weight, backward: gradient), out-edges (ring row, weight, byte offset
// of the step; backward), the slice's G.
template <int VB>
static size_t rs_warp_ints(int cap, bool backward) {
  return backward ? (size_t)8 * cap + 32 * VB : (size_t)3 * cap;
}

struct RsEdges {
  int *ibase, *id;
  float* iw;
  float* iacc;
  int* orow;     // d * N + post, delay-1 synapses first
  float2* pair;  // (byte offset in the ring, weight)
  float* g;
  int nin, nout, none;
};

// 32 x 32 bit transpose over the lanes: bit p of the result in lane b is bit
// b of x in lane p.
__device__ __forceinline__ unsigned bit_transpose(unsigned x, int lane) {
  unsigned y = __shfl_xor_sync(0xffffffffu, x, 16);
  x = (lane & 16) ? __byte_perm(x, y, 0x3276) : __byte_perm(x, y, 0x5410);
  y = __shfl_xor_sync(0xffffffffu, x, 8);
  x = (lane & 8) ? __byte_perm(x, y, 0x3715) : __byte_perm(x, y, 0x6240);
#pragma unroll
  for (int j = 4; j >= 1; j >>= 1) {
    const unsigned m = j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    y = __shfl_xor_sync(0xffffffffu, x, j);
    y = __funnelshift_l(y, y, (lane & j) ? 32 - j : j);
    const unsigned keep = (lane & j) ? ~m : m;
    x = (x & keep) | (y & ~keep);
  }
  return x;
}

// The in-edges of neuron j, whole groups of 32.
template <int VB>
__device__ __forceinline__ void rs_stage_in(const BpArgs& a, int j, int sl, bool acc, RsEdges& we) {
  const int lane = threadIdx.x & 31;
  const int c0 = a.col_ptr[j];
  we.nin = a.col_ptr[j + 1] - c0;
  for (int g = 0; g < we.nin; g += 32) {
    const int e = g + lane;
    const bool ok = e < we.nin;
    const int d = ok ? a.in_d[c0 + e] : INT_MAX;
    we.id[g + lane] = d;
    we.ibase[g + lane] = ok ? (a.in_pre[c0 + e] - d * a.N) * a.KBs + sl * VB : 0;
    we.iw[g + lane] = ok ? a.w[a.in_eidx[c0 + e]] : 0.f;
    if (acc) we.iacc[g + lane] = 0.f;
  }
  __syncwarp();
}

// Spike words of this lane's edge of group g for step t (0 before step d);
// row: a.bits + t * N * KBs, nw: the slice's words (at most VB).
template <int VB>
__device__ __forceinline__ void rs_words(const uint32_t* row, const RsEdges& we, int g, int t, int nw,
                                         uint32_t (&w)[VB]) {
  const int at = g * 32 + (threadIdx.x & 31);
  const bool ok = we.id[at] <= t;
  const uint32_t* wp = row + we.ibase[at];
#pragma unroll
  for (int k = 0; k < VB; ++k) w[k] = ok && k < nw ? wp[k] : 0u;
}

// acc[k] += val[i] for every set bit i < n of x[k], in order (val: shared
// memory, 16-byte aligned, readable in whole quads).
template <int VB>
__device__ __forceinline__ void rs_add_bits(const float* val, int n, const uint32_t (&x)[VB], float (&acc)[VB]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (4 * q >= n) break;
    const float4 f = *reinterpret_cast<const float4*>(val + 4 * q);
#pragma unroll
    for (int k = 0; k < VB; ++k) {
      if (x[k] & (1u << (4 * q))) acc[k] = __fadd_rn(acc[k], f.x);
      if (x[k] & (2u << (4 * q))) acc[k] = __fadd_rn(acc[k], f.y);
      if (x[k] & (4u << (4 * q))) acc[k] = __fadd_rn(acc[k], f.z);
      if (x[k] & (8u << (4 * q))) acc[k] = __fadd_rn(acc[k], f.w);
    }
  }
}

// The delivered current of step t; w0: the words of the first groups.
template <int VB>
__device__ __forceinline__ void rs_current(const uint32_t* row, const RsEdges& we, int t, int nw,
                                           uint32_t (&w0)[kRsGroups<VB>][VB], float (&acc)[VB]) {
  constexpr int G = kRsGroups<VB>;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < VB; ++k) acc[k] = 0.f;
  for (int e0 = 0; e0 < we.nin; e0 += 32 * G) {
    if (e0 > 0) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (e0 + 32 * g < we.nin) rs_words<VB>(row, we, e0 / 32 + g, t, nw, w0[g]);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int n = we.nin - e0 - 32 * g;
      if (n <= 0) break;
#pragma unroll
      for (int k = 0; k < VB; ++k) w0[g][k] = bit_transpose(w0[g][k], lane);
      rs_add_bits<VB>(we.iw + e0 + 32 * g, n, w0[g], acc);
    }
  }
}

template <int VB, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_res_forward(BpArgs a) {
  extern __shared__ __align__(16) float sm_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int item = a.even ? (int)(blockIdx.x * (blockDim.x >> 5)) + warp : warp * (int)gridDim.x + (int)blockIdx.x;
  const bool on = item < a.N * a.SL;
  const int j = on ? item % a.N : 0, sl = on ? item / a.N : 0;
  const int N = a.N, B = a.B, b0 = sl * 32 * VB + lane;
  const int nw = min(VB, a.KBs - sl * VB);        // this slice's words
  const int row_w = N * a.KBs;                    // words of a step
  uint32_t* row = a.bits;                         // the step's words
  const size_t NB = (size_t)N * B;
  size_t plane = (size_t)j * B + b0, save = plane; // this warp's place in the step's / checkpoint's plane
  int left = a.K;                                 // steps to the next checkpoint
  RsEdges we{};
  we.ibase = reinterpret_cast<int*>(sm_all) + (size_t)warp * 3 * a.res_cap;
  we.id = we.ibase + a.res_cap;
  we.iw = reinterpret_cast<float*>(we.id + a.res_cap);
  if (on) rs_stage_in<VB>(a, j, sl, false, we);
  float v[VB], x_ext[VB];
  constexpr int G = kRsGroups<VB>;
  uint32_t w0[G][VB];
#pragma unroll
  for (int k = 0; k < VB; ++k) {
    v[k] = 0.f;
    x_ext[k] = on && b0 + 32 * k < B ? a.ext[(size_t)j * B + b0 + 32 * k] : 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) w0[g][k] = 0u;
  }
  unsigned target = a.stall;
  for (int t = 0; t < a.T; ++t) {
    float vp[VB], s[VB];
    if (on) {
      float acc[VB];
      rs_current<VB>(row, we, t, nw, w0, acc);
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        vp[k] = __fadd_rn(__fadd_rn(__fmul_rn(a.decay, v[k]), acc[k]), x_ext[k]);
        s[k] = __fsub_rn(vp[k], a.thr) >= 0.f ? 1.f : 0.f;
        v[k] = __fmul_rn(vp[k], __fsub_rn(1.f, s[k]));
        const unsigned m = __ballot_sync(0xffffffffu, b0 + 32 * k < B && s[k] != 0.f);
        if (lane == 0 && k < nw) row[j * a.KBs + sl * VB + k] = m;
      }
    }
    target += gridDim.x;
    grid_arrive(&a.ctl[0]);
    if (on) {
      const bool keep = a.K == 0 || --left == 0 || t + 1 == a.T;
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        if (b0 + 32 * k >= B) continue;
        a.spikes[plane + 32 * k] = s[k];
        if (keep) a.vsaved[save + 32 * k] = a.K == 0 ? vp[k] : v[k];
        if (t + 1 < a.T) x_ext[k] = a.ext[plane + NB + 32 * k];
      }
      if (keep) {
        save += NB;
        left = a.K;
      }
      plane += NB;
      row += row_w;
      // the next step's words of delay 2 and more are final already
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (32 * g < we.nin && we.id[32 * g + lane] > 1) rs_words<VB>(row, we, g, t + 1, nw, w0[g]);
    }
    if (!grid_wait(&a.ctl[0], target, a.err, a.wait_ns)) return;
    if (on && t + 1 < a.T) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (32 * g < we.nin && we.id[32 * g + lane] == 1) rs_words<VB>(row, we, g, t + 1, nw, w0[g]);
    }
  }
}

template <int VB, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_res_backward(BpArgs a) {
  typedef typename VecOf<VB>::T Vec;
  extern __shared__ __align__(16) float sm_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int item = a.even ? (int)(blockIdx.x * (blockDim.x >> 5)) + warp : warp * (int)gridDim.x + (int)blockIdx.x;
  const bool on = item < a.N * a.SL;
  const int j = on ? item % a.N : 0, sl = on ? item / a.N : 0;
  const int N = a.N, B = a.B, T = a.T, R = a.R, K = a.K, cap = a.res_cap;
  const int bf = sl * 32 * VB + lane, bb = sl * 32 * VB + VB * lane;  // forward / vector sample order
  const int nw = min(VB, a.KBs - sl * VB);                            // this slice's words
  const int row_w = N * a.KBs, ring_n = R * N;
  RsEdges we{};
  {
    float* p = sm_all + (size_t)warp * (8 * cap + 32 * VB);
    we.pair = reinterpret_cast<float2*>(p);
    we.g = p + 2 * cap;
    we.ibase = reinterpret_cast<int*>(we.g + 32 * VB);
    we.id = we.ibase + cap;
    we.iw = reinterpret_cast<float*>(we.id + cap);
    we.iacc = we.iw + cap;
    we.orow = reinterpret_cast<int*>(we.iacc + cap);
  }
  if (on) rs_stage_in<VB>(a, j, sl, true, we);
  // out-edges, those of delay 1 first, each part in CSR order, with `left` steps
  // to the end: weight 0 for those that reach beyond it
  auto stage_out = [&](int left) {
    const int r0 = a.row_ptr[j], n = a.row_ptr[j + 1] - r0;
    we.nout = n;
    int at = 0;
    for (int part = 0; part < 2; ++part) {
      for (int e0 = 0; e0 < n; e0 += 32) {
        const int e = e0 + lane;
        const int d = e < n ? a.out_d[r0 + e] : 0;
        const bool mine = e < n && (d == 1) == (part == 0);
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine) {
          const int q = at + __popc(m & ((1u << lane) - 1u));
          we.orow[q] = d * N + a.out_post[r0 + e];
          we.pair[q] = make_float2(0.f, d < left ? a.w[r0 + e] : 0.f);
        }
        at += __popc(m);
      }
      if (part == 0) we.none = at;
    }
    __syncwarp();
  };
  const unsigned row_b = (unsigned)a.Bp * 4u;  // bytes of a ring row
  const char* ring_l = reinterpret_cast<const char*>(a.ring) + (size_t)bb * 4;
  auto one = [&](int e, float (&acc)[VB]) {
    const float2 p = we.pair[e];
    const Vec x = *reinterpret_cast<const Vec*>(ring_l + __float_as_uint(p.x));
#pragma unroll
    for (int k = 0; k < VB; ++k) acc[k] = __fmaf_rn(p.y, reinterpret_cast<const float*>(&x)[k], acc[k]);
  };
  // acc += the gradients of out-edges [e0, e1) at step t, in that order
  // (base: the step's slot * N)
  auto gather = [&](int base, int e0, int e1, float (&acc)[VB]) {
    for (int e = e0 + lane; e < e1; e += 32) {
      int r = base + we.orow[e];
      if (r >= ring_n) r -= ring_n;
      we.pair[e].x = __uint_as_float((unsigned)r * row_b);
    }
    __syncwarp();
    constexpr int U = VB == 4 ? 4 : 8;
    int e = e0;
    for (; e < e1 && (e & 1); ++e) one(e, acc);
    for (; e + U <= e1; e += U) {
      Vec x[U];
      float w[U];
#pragma unroll
      for (int u = 0; u < U; u += 2) {
        const float4 p = *reinterpret_cast<const float4*>(&we.pair[e + u]);
        w[u] = p.y;
        w[u + 1] = p.w;
        x[u] = *reinterpret_cast<const Vec*>(ring_l + __float_as_uint(p.x));
        x[u + 1] = *reinterpret_cast<const Vec*>(ring_l + __float_as_uint(p.z));
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < VB; ++k) acc[k] = __fmaf_rn(w[u], reinterpret_cast<const float*>(&x[u])[k], acc[k]);
    }
    for (; e < e1; ++e) one(e, acc);
    __syncwarp();
  };
  // pre-reset potentials of segment sg from its checkpoint and the stored spikes
  auto recompute = [&](int sg) {
    const int t0 = sg * K, t1 = min(T, t0 + K);
    const uint32_t* row = a.bits + (size_t)t0 * row_w;
    const float* ext = a.ext + ((size_t)t0 * N + j) * B + bf;
    float* seg = a.seg + (size_t)j * a.Bp + bf;  // rows as the ring's
    float v[VB];
#pragma unroll
    for (int k = 0; k < VB; ++k)
      v[k] = sg > 0 && bf + 32 * k < B ? a.vsaved[((size_t)(sg - 1) * N + j) * B + bf + 32 * k] : 0.f;
    for (int t = t0; t < t1; ++t) {
      float acc[VB], x_ext[VB];
      uint32_t w0[kRsGroups<VB>][VB];
#pragma unroll
      for (int g = 0; g < kRsGroups<VB>; ++g)
        if (32 * g < we.nin) rs_words<VB>(row, we, g, t, nw, w0[g]);
#pragma unroll
      for (int k = 0; k < VB; ++k)
        x_ext[k] = bf + 32 * k < B ? ext[32 * k] : 0.f;
      rs_current<VB>(row, we, t, nw, w0, acc);
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        const float vp = __fadd_rn(__fadd_rn(__fmul_rn(a.decay, v[k]), acc[k]), x_ext[k]);
        const float s = __fsub_rn(vp, a.thr) >= 0.f ? 1.f : 0.f;
        v[k] = __fmul_rn(vp, __fsub_rn(1.f, s));
        if (bf + 32 * k < B) seg[32 * k] = vp;
      }
      row += row_w;
      ext += (size_t)N * B;
      seg += (size_t)N * a.Bp;
    }
    __syncwarp();
  };
  float gv[VB], gs[VB], vp[VB];
#pragma unroll
  for (int k = 0; k < VB; ++k) gv[k] = gs[k] = vp[k] = 0.f;
  // what step t (place kp of its segment, slot base `base`) needs that is
  // final before its barrier
  int kp = K > 0 ? (T - 1) % K : 0, base = ((T - 1) % R) * N;
  auto prepare = [&](int t) {
    if (T - t <= R) stage_out(T - t);  // (the last time with every weight)
    if (K > 0 && (t == T - 1 || kp == K - 1)) recompute(t / K);
    const size_t plane = ((size_t)t * N + j) * B + bb;
#pragma unroll
    for (int k = 0; k < VB; ++k) {
      gs[k] = bb + k < B ? a.gspk[plane + k] : 0.f;
      vp[k] = K == 0 ? (bb + k < B ? a.vsaved[plane + k] : 0.f)
                     : a.seg[((size_t)kp * N + j) * a.Bp + bb + k];
    }
    gather(base, we.none, we.nout, gs);
  };
  unsigned target = a.stall;
  if (on) prepare(T - 1);
  for (int t = T - 1; t >= 0; --t) {
    float g[VB];
    if (on) {
      float g1[VB];
#pragma unroll
      for (int k = 0; k < VB; ++k) g1[k] = 0.f;
      gather(base, 0, we.none, g1);
      Vec out;
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        const float x = __fsub_rn(vp[k], a.thr);
        const float den = __fadd_rn(1.f, __fmul_rn(a.slope, fabsf(x)));
        const float s = x >= 0.f ? 1.f : 0.f;
        const float sg = __fdiv_rn(1.f, __fmul_rn(den, den));
        const float gst = __fsub_rn(__fadd_rn(gs[k], g1[k]), __fmul_rn(gv[k], vp[k]));
        g[k] = __fadd_rn(__fmul_rn(gv[k], __fsub_rn(1.f, s)), __fmul_rn(gst, sg));
        gv[k] = __fmul_rn(a.decay, g[k]);
        if (bb + k >= B) g[k] = gv[k] = 0.f;
        reinterpret_cast<float*>(&out)[k] = g[k];
      }
      if (bb < B) *reinterpret_cast<Vec*>(a.ring + (size_t)(base + j) * a.Bp + bb) = out;
    }
    target += gridDim.x;
    grid_arrive(&a.ctl[0]);
    if (on) {
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        we.g[VB * lane + k] = g[k];
        if (a.gext && bb + k < B) a.gext[((size_t)t * N + j) * B + bb + k] = g[k];
      }
      __syncwarp();
      // dL/dw of this lane's in-edges: the sum of G over the samples whose pre
      // fired at t - d
      const int ng = (we.nin + 31) >> 5;
      const uint32_t* row = a.bits + (size_t)t * row_w;
      for (int q0 = 0; q0 < ng; q0 += kRsGroups<VB>) {
        uint32_t w[kRsGroups<VB>][VB];
#pragma unroll
        for (int q = 0; q < kRsGroups<VB>; ++q)
          if (q0 + q < ng) rs_words<VB>(row, we, q0 + q, t, nw, w[q]);
#pragma unroll
        for (int q = 0; q < kRsGroups<VB>; ++q) {
          if (q0 + q >= ng) break;
          float c[1] = {0.f};
#pragma unroll
          for (int k = 0; k < VB; ++k) {
            const uint32_t wk[1] = {w[q][k]};
            rs_add_bits<1>(we.g + 32 * k, 32, wk, c);
          }
          if (c[0] != 0.f)
            we.iacc[32 * (q0 + q) + lane] = __fadd_rn(we.iacc[32 * (q0 + q) + lane], c[0]);
        }
      }
      __syncwarp();
      base = base == 0 ? ring_n - N : base - N;
      kp = kp == 0 ? K - 1 : kp - 1;
      if (t > 0) prepare(t - 1);
    }
    if (!grid_wait(&a.ctl[0], target, a.err, a.wait_ns)) return;
  }
  if (on) {
    const int c0 = a.col_ptr[j];
    for (int e = lane; e < we.nin; e += 32)
      a.part[(size_t)sl * a.S + a.in_eidx[c0 + e]] = we.iacc[e];
  }
}

using BpKernel = void (*)(BpArgs);

// Co-resident warps of a launch of kern with smem bytes per block.
static int resident_warps(BpKernel kern, size_t smem, int sm_count) {
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBpThreads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm * sm_count * (kBpThreads / 32);
}

static int coop_launch(BpKernel kern, const BpArgs& a, int sm_count, size_t smem, cudaStream_t st) {
  SNCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  SNCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBpThreads, smem));
  if (per_sm < 1) {
    set_error("bptt kernel does not fit on an SM");
    return SNC_B200_EUNSUPPORTED;
  }
  const int warps_needed = a.N;
  const int blocks = std::max(1, std::min(per_sm * sm_count, (warps_needed + 7) / 8));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kBpThreads);
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

// A launch with staged edges (smooth spikes, a.res_cap > 0) when one warp per
// neuron can be co-resident with them, else the global-memory form.
template <int KB>
static int dispatch(bool forward, bool smooth, BpArgs a, int sm, cudaStream_t st) {
  const size_t smem = forward ? 0 : (size_t)(kBpThreads / 32) * 32 * KB * sizeof(float);
  if (smooth && a.res_cap > 0) {
    const size_t smem_r = smem + (size_t)(kBpThreads / 32) * 8 * a.res_cap * sizeof(int);
    BpKernel kr = forward ? k_bptt_forward<KB, true, true> : k_bptt_backward<KB, true, true, false>;
    if (resident_warps(kr, smem_r, sm) >= a.N) return coop_launch(kr, a, sm, smem_r, st);
  }
  a.res_cap = 0;
  BpKernel k = forward ? (smooth ? k_bptt_forward<KB, true, false> : k_bptt_forward<KB, false, false>)
                       : (smooth ? k_bptt_backward<KB, true, false, false>
                          : a.split ? k_bptt_backward<KB, false, false, true>
                                    : k_bptt_backward<KB, false, false, false>);
  return coop_launch(k, a, sm, smem, st);
}

constexpr int kMaxWords = 8;  // 32-sample words of a batch that any form takes

// Batch slices.  a.split: the resident launches can take this net and batch --
// binary spikes, all warps co-resident (32 to an SM) with their edges in shared
// memory (cap per direction; 0: too many), indexes of 32 bits -- in slices of
// the fewest words (more warps hide more latency: core of 1808 neurons, 128
// samples, 1 slice of 4 words to 2 of 2).  The global-memory form then sums in
// their order, whether or not they are on.  Everything else is one slice, summed
// in edge order: a sum per slice and two per gather cost the general form of 512
// neurons of degree 300 at 128 samples 3.4 against 2.3 ms.
static void pick_slices(BpArgs& a, int cap, int sm) {
  a.KBs = (a.B + 31) / 32;
  a.SL = 1;
  a.split = 0;
  if (a.smooth || cap <= 0 || a.KBs > kMaxWords) return;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (((long long)a.T + a.R) * a.N * a.KBs >= INT_MAX || (long long)a.R * a.N >= INT_MAX / 2) return;
  for (int lg = 0; lg <= 2; ++lg) {
    const int vb = 1 << lg, sl = (a.KBs + vb - 1) / vb;
    const long long items = (long long)a.N * sl, warps = (items + sm - 1) / sm;
    const size_t ints = lg == 0 ? rs_warp_ints<1>(cap, true) : lg == 1 ? rs_warp_ints<2>(cap, true) : rs_warp_ints<4>(cap, true);
    if (warps > 32 || ints * 4 * warps + 1024 > (size_t)optin ||
        ((long long)a.R * a.N + 1) * sl * vb * 128 > (long long)UINT_MAX)
      continue;
    a.split = 1;
    a.VB = vb;
    a.VB_log = lg;
    a.SL = sl;
    const int unit = a.B < 8 ? vb : 8;  // whole 32-byte sectors, where rows have any
    a.Bp = (a.B + unit - 1) / unit * unit;
    return;
  }
}

// This launch is a resident one.
static bool rs_takes(const BpArgs& a) { return a.split && a.res_cap > 0; }

template <int VB>
static int rs_launch(bool forward, const BpArgs& a, int sm, cudaStream_t st) {
  const long long items = (long long)a.N * a.SL;
  const int warps = (int)((items + sm - 1) / sm);
  const int grid = (int)((items + warps - 1) / warps);
  const size_t smem = rs_warp_ints<VB>(a.res_cap, !forward) * 4 * warps;
  // fewer warps leave each more registers
  BpKernel kern = forward ? (warps <= 24 ? k_res_forward<VB, 768> : warps <= 28 ? k_res_forward<VB, 896> : k_res_forward<VB, 1024>)
                          : (warps <= 24 ? k_res_backward<VB, 768> : warps <= 28 ? k_res_backward<VB, 896> : k_res_backward<VB, 1024>);
  SNCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * warps);
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

static int launch(bool forward, bool smooth, const BpArgs& a, int sm, cudaStream_t st) {
  if (rs_takes(a))
    return a.VB == 1 ? rs_launch<1>(forward, a, sm, st)
           : a.VB == 2 ? rs_launch<2>(forward, a, sm, st) : rs_launch<4>(forward, a, sm, st);
  const int KB = a.KBs;
  if (KB <= 1) return dispatch<1>(forward, smooth, a, sm, st);
  if (KB <= 2) return dispatch<2>(forward, smooth, a, sm, st);
  if (KB <= 4) return dispatch<4>(forward, smooth, a, sm, st);
  if (KB <= kMaxWords) return dispatch<8>(forward, smooth, a, sm, st);
  set_error("bptt: batch > 256");
  return SNC_B200_EUNSUPPORTED;
}

template <typename T>
static int grow(T** p, size_t* cap, size_t n) {
  if (*p && *cap >= n) return SNC_B200_OK;
  dev_free(*p);
  *p = nullptr;
  *cap = 0;
  int rc = dev_alloc(p, n);
  if (!rc) *cap = n;
  return rc;
}

// Edges per direction a resident launch stages per warp (0: too many).
static int res_cap(const snc_b200_bptt* h) {
  if (h->max_deg > kResCapMax) return 0;
  return std::max(32, (h->max_deg + 31) / 32 * 32);
}

// Arguments of a forward launch over handle h (both forward entry points).
static BpArgs forward_args(const snc_b200_bptt* h, const float* w, const float* ext, int T, int B,
                           float threshold, float decay, float slope, int ckpt_every, int smooth,
                           float* spikes, uint32_t* spike_bits, float* v_saved) {
  BpArgs a{};
  a.N = h->N; a.S = h->S; a.R = h->R; a.T = T; a.B = B; a.K = ckpt_every; a.smooth = smooth;
  a.thr = threshold; a.decay = decay; a.slope = slope;
  a.row_ptr = h->row_ptr; a.out_post = h->out_post; a.out_d = h->out_d; a.col_ptr = h->col_ptr;
  a.in_pre = h->in_pre; a.in_d = h->in_d; a.in_eidx = h->in_eidx;
  a.w = w; a.ext = ext; a.spikes = spikes; a.bits = spike_bits; a.vsaved = v_saved;
  a.res_cap = h->resident ? res_cap(h) : 0;
  a.even = h->even;
  pick_slices(a, res_cap(h), h->sm_count);
  const WaitCtl wc = take_wait_ctl(true);
  a.wait_ns = wc.ns;
  a.stall = wc.stall;
  return a;
}

static int check_err(snc_b200_bptt* h, cudaStream_t st) {
  int err = 0;
  SNCB_CUDA(cudaMemcpyAsync(&err, h->err, sizeof(int), cudaMemcpyDeviceToHost, st));
  SNCB_CUDA(cudaStreamSynchronize(st));
  if (err) {
    set_error("bptt: device barrier timed out");
    return err;
  }
  return SNC_B200_OK;
}

}  // namespace sncb

using namespace sncb;

// Leaky integration along time of a [T][n] tensor: y[t] = decay * y[t-1] +
// x[t] (reverse: from the last step backwards, y[t] = decay * y[t+1] + x[t]),
// each product and sum rounded separately like the step-by-step loop of the
// readouts (shd_model.py:139-140, lm.py:90); the reverse form is its
// gradient.  A thread takes W neighbouring columns, the loads of several steps at
// once.  Four columns where there are many: 268 MB in and out (4096 x 64 columns,
// 256 steps) in 83 us, the rate of a plain copy, 111 with a 4-byte load a step.
// One column where there are few, and then a thread's own chain of steps is what
// counts: it requests 16 steps while it adds the 16 before (64 columns, 1000
// steps: 20 us, 69 with eight requested behind each other's sums).
template <int W>
__global__ void k_leaky_scan(const float* __restrict__ x, float* __restrict__ y, int T, long long n,
                             float decay, int reverse) {
  constexpr int U = W == 1 ? 16 : 8;
  struct alignas(4 * W) Vec {
    float v[W];
  };
  const long long step = reverse ? -n : n, first = reverse ? (T - 1) * n : 0;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n / W;
       j += (long long)gridDim.x * blockDim.x) {
    const float* p = x + first + j * W;
    float* q = y + first + j * W;
    float acc[W];
#pragma unroll
    for (int i = 0; i < W; ++i) acc[i] = 0.f;
    auto get = [&](Vec (&s)[U]) {
#pragma unroll
      for (int u = 0; u < U; ++u, p += step) s[u] = *reinterpret_cast<const Vec*>(p);
    };
    auto put = [&](Vec& s) {
#pragma unroll
      for (int i = 0; i < W; ++i) s.v[i] = acc[i] = __fadd_rn(__fmul_rn(decay, acc[i]), s.v[i]);
      *reinterpret_cast<Vec*>(q) = s;
      q += step;
    };
    int left = T;
    Vec in[U];
    if (W == 1 && left >= U) get(in);
    for (; left >= (W == 1 ? 2 * U : U); left -= U) {
      Vec next[U];
      get(W == 1 ? next : in);
#pragma unroll
      for (int u = 0; u < U; ++u) put(in[u]);
      if (W == 1)
#pragma unroll
        for (int u = 0; u < U; ++u) in[u] = next[u];
    }
    if (W == 1 && left >= U) {
#pragma unroll
      for (int u = 0; u < U; ++u) put(in[u]);
      left -= U;
    }
    for (; left > 0; --left, p += step) {
      Vec s = *reinterpret_cast<const Vec*>(p);
      put(s);
    }
  }
}

// out[t][i][j] = in[t * st_t + i + j * st_j]: the batch-innermost layout of
// the BPTT kernels and torch's [T][B][N] (or a view of it with unit stride
// along N) into each other, through 64 x 64 shared-memory tiles so that both
// the reads (along i) and the writes (along j) are coalesced, 16 bytes a thread
// and access where the rows allow it (VI, VO: all rows of that side start on
// 16 bytes).  Four loads a thread in flight; 268 MB in and
// out took 180 us with 4 bytes an access, 78 so.
constexpr int kTrTile = 64;

template <bool VI, bool VO>
__global__ void __launch_bounds__(256) k_transpose_tile(const float* __restrict__ in, float* __restrict__ out,
                                                        int I, int J, long long st_t, long long st_j) {
  __shared__ float tile[kTrTile][kTrTile + 1];  // [j][i]
  const int i0 = blockIdx.x * kTrTile, j0 = blockIdx.y * kTrTile;
  const long long t = blockIdx.z;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float* src = in + t * st_t;
  float* dst = out + t * (long long)I * J;
  float4 f[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int j = j0 + ty + 16 * k, i = i0 + 4 * tx;
    f[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j >= J) continue;
    const float* p = src + (long long)j * st_j + i;
    if (VI && i + 3 < I) {
      f[k] = *reinterpret_cast<const float4*>(p);
    } else {
      if (i < I) f[k].x = p[0];
      if (i + 1 < I) f[k].y = p[1];
      if (i + 2 < I) f[k].z = p[2];
      if (i + 3 < I) f[k].w = p[3];
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float* q = &tile[ty + 16 * k][4 * tx];
    q[0] = f[k].x;
    q[1] = f[k].y;
    q[2] = f[k].z;
    q[3] = f[k].w;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int ii = ty + 16 * k, i = i0 + ii, j = j0 + 4 * tx;
    if (i >= I) continue;
    const float4 v = make_float4(tile[4 * tx][ii], tile[4 * tx + 1][ii], tile[4 * tx + 2][ii], tile[4 * tx + 3][ii]);
    float* p = dst + (long long)i * J + j;
    if (VO && j + 3 < J) {
      *reinterpret_cast<float4*>(p) = v;
    } else {
      if (j < J) p[0] = v.x;
      if (j + 1 < J) p[1] = v.y;
      if (j + 2 < J) p[2] = v.z;
      if (j + 3 < J) p[3] = v.w;
    }
  }
}

extern "C" {

int snc_b200_bptt_create(int32_t N, int32_t S, const int32_t* row_ptr, const int32_t* post,
                         const int32_t* delays, snc_b200_bptt** out) {
  if (!out || N <= 0 || S < 0 || !row_ptr || (S > 0 && (!post || !delays)) || row_ptr[0] != 0 ||
      row_ptr[N] != S) {
    set_error("bptt_create: bad graph");
    return SNC_B200_EINVAL;
  }
  for (int i = 0; i < N; ++i)
    if (row_ptr[i] > row_ptr[i + 1]) { set_error("bptt_create: row_ptr not monotone"); return SNC_B200_EINVAL; }
  int D = 1;
  for (int e = 0; e < S; ++e) {
    if (post[e] < 0 || post[e] >= N || delays[e] < 1) { set_error("bptt_create: bad edge"); return SNC_B200_EINVAL; }
    D = std::max(D, delays[e]);
  }
  *out = nullptr;
  auto* h = new snc_b200_bptt();
  h->N = N;
  h->S = S;
  h->D = D;
  h->R = D + 1;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, dev);
  // incoming lists in ascending CSR edge order
  std::vector<int> col_ptr(N + 1, 0), in_pre(std::max(1, S)), in_d(std::max(1, S)), in_eidx(std::max(1, S));
  for (int e = 0; e < S; ++e) col_ptr[post[e] + 1]++;
  for (int j = 0; j < N; ++j)
    h->max_deg = std::max({h->max_deg, col_ptr[j + 1], row_ptr[j + 1] - row_ptr[j]});
  for (int j = 0; j < N; ++j) col_ptr[j + 1] += col_ptr[j];
  // (a quarter above the mean: a random net of 64 synapses a neuron stays
  // within a tenth; a layer without synapses in one direction is at 3/2)
  h->even = true;
  for (int j = 0; j < N && h->even; j += 32) {
    const int k = std::min(N, j + 32);
    const double edges = (double)(col_ptr[k] - col_ptr[j]) + (row_ptr[k] - row_ptr[j]);
    h->even = edges * N <= 1.25 * 2.0 * S * 32;
  }
  std::vector<int> fill(col_ptr.begin(), col_ptr.end() - 1);
  for (int i = 0; i < N; ++i)
    for (int e = row_ptr[i]; e < row_ptr[i + 1]; ++e) {
      const int q = fill[post[e]]++;
      in_pre[q] = i;
      in_d[q] = delays[e];
      in_eidx[q] = e;
    }
  int rc = SNC_B200_OK;
  if (!rc) rc = dev_upload(&h->row_ptr, row_ptr, (size_t)N + 1);
  if (!rc) rc = dev_upload(&h->out_post, post, (size_t)std::max(1, S));
  if (!rc) rc = dev_upload(&h->out_d, delays, (size_t)std::max(1, S));
  if (!rc) rc = dev_upload(&h->col_ptr, col_ptr.data(), col_ptr.size());
  if (!rc) rc = dev_upload(&h->in_pre, in_pre.data(), in_pre.size());
  if (!rc) rc = dev_upload(&h->in_d, in_d.data(), in_d.size());
  if (!rc) rc = dev_upload(&h->in_eidx, in_eidx.data(), in_eidx.size());
  if (!rc) rc = dev_alloc(&h->ctl, 4);
  if (!rc) rc = dev_alloc(&h->err, 1);
  if (rc) {
    snc_b200_bptt_release(h);
    return rc;
  }
  *out = h;
  return SNC_B200_OK;
}

int snc_b200_bptt_set_resident(snc_b200_bptt* h, int32_t enable) {
  if (!h) {
    set_error("bptt_set_resident: null handle");
    return SNC_B200_EINVAL;
  }
  h->resident = enable != 0;
  return SNC_B200_OK;
}

int snc_b200_bptt_release(snc_b200_bptt* h) {
  if (!h) return SNC_B200_OK;
  const PoolBatch batch;
  for (void* p : {(void*)h->row_ptr, (void*)h->out_post, (void*)h->out_d, (void*)h->col_ptr,
                  (void*)h->in_pre, (void*)h->in_d, (void*)h->in_eidx, (void*)h->v, (void*)h->gv,
                  (void*)h->gcur, (void*)h->seg, (void*)h->part, (void*)h->ctl, (void*)h->err})
    dev_free(p);
  delete h;
  return SNC_B200_OK;
}

int snc_b200_bptt_forward(snc_b200_bptt* h, const float* w, const float* ext, int32_t T, int32_t B,
                          float threshold, float decay, float slope, int32_t ckpt_every,
                          int32_t smooth, float* spikes, uint32_t* spike_bits, float* v_saved,
                          void* stream) {
  if (!h || !w || !ext || !spikes || !v_saved || T < 1 || B < 1 || ckpt_every < 0 ||
      (!smooth && !spike_bits)) {
    set_error("bptt_forward: bad argument");
    return SNC_B200_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t NB = (size_t)h->N * B;
  int rc = grow(&h->v, &h->v_cap, NB);
  if (rc) return rc;
  BpArgs a = forward_args(h, w, ext, T, B, threshold, decay, slope, ckpt_every, smooth, spikes,
                          spike_bits, v_saved);
  a.v = h->v;
  a.ctl = h->ctl; a.err = h->err;
  SNCB_CUDA(cudaMemsetAsync(h->ctl, 0, 16, st));
  SNCB_CUDA(cudaMemsetAsync(h->err, 0, 4, st));
  if ((rc = launch(true, smooth != 0, a, h->sm_count, st))) return rc;
  return check_err(h, st);
}

int snc_b200_bptt_backward(snc_b200_bptt* h, const float* w, const float* ext, int32_t T, int32_t B,
                           float threshold, float decay, float slope, int32_t ckpt_every,
                           int32_t smooth, const float* spikes, const uint32_t* spike_bits,
                           const float* v_saved, const float* grad_spikes, float* grad_w,
                           float* grad_ext, void* stream) {
  if (!h || !w || !ext || !spikes || !v_saved || !grad_spikes || !grad_w || T < 1 || B < 1 ||
      ckpt_every < 0 || (!smooth && !spike_bits)) {
    set_error("bptt_backward: bad argument");
    return SNC_B200_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t NB = (size_t)h->N * B;
  int rc;
  BpArgs a{};
  a.N = h->N; a.S = h->S; a.R = h->R; a.T = T; a.B = B; a.K = ckpt_every; a.smooth = smooth;
  a.thr = threshold; a.decay = decay; a.slope = slope;
  a.row_ptr = h->row_ptr; a.out_post = h->out_post; a.out_d = h->out_d; a.col_ptr = h->col_ptr;
  a.in_pre = h->in_pre; a.in_d = h->in_d; a.in_eidx = h->in_eidx;
  a.w = w; a.ext = ext; a.spikes = const_cast<float*>(spikes);
  a.bits = const_cast<uint32_t*>(spike_bits); a.vsaved = const_cast<float*>(v_saved);
  a.gspk = grad_spikes; a.gext = grad_ext;
  a.ctl = h->ctl; a.err = h->err;
  a.res_cap = h->resident ? res_cap(h) : 0;
  a.even = h->even;
  pick_slices(a, res_cap(h), h->sm_count);
  const bool rs = rs_takes(a);
  // the resident form keeps its state in registers; its lanes beyond the batch
  // read behind the last rows
  const size_t rows = rs ? (size_t)h->N * a.Bp : NB, behind = rs ? (size_t)a.SL * a.VB * 32 : 0;
  if (!rs && (rc = grow(&h->v, &h->v_cap, NB))) return rc;
  if (!rs && (rc = grow(&h->gv, &h->gv_cap, NB))) return rc;
  if ((rc = grow(&h->gcur, &h->gcur_cap, (size_t)h->R * rows + behind))) return rc;
  if (ckpt_every > 0 && (rc = grow(&h->seg, &h->seg_cap, (size_t)ckpt_every * rows + behind))) return rc;
  if (a.SL > 1 && (rc = grow(&h->part, &h->part_cap, (size_t)a.SL * std::max(1, h->S)))) return rc;
  a.v = h->v; a.gv = h->gv; a.gcur = h->gcur; a.ring = h->gcur; a.seg = h->seg;
  a.part = a.SL > 1 ? h->part : grad_w;
  const WaitCtl wc = take_wait_ctl(true);
  a.wait_ns = wc.ns;
  a.stall = wc.stall;
  SNCB_CUDA(cudaMemsetAsync(h->ctl, 0, 16, st));
  SNCB_CUDA(cudaMemsetAsync(h->err, 0, 4, st));
  if (rs) SNCB_CUDA(cudaMemsetAsync(a.ring, 0, (size_t)h->R * rows * sizeof(float), st));
  else SNCB_CUDA(cudaMemsetAsync(a.part, 0, (size_t)a.SL * h->S * sizeof(float), st));
  if ((rc = launch(false, smooth != 0, a, h->sm_count, st))) return rc;
  if (a.SL > 1 && h->S > 0) {
    k_sum_slices<<<std::min((h->S + 255) / 256, h->sm_count * 8), 256, 0, st>>>(h->S, a.SL, a.part, grad_w);
    SNCB_CUDA(cudaGetLastError());
  }
  return check_err(h, st);
}

int snc_b200_leaky_scan(const float* x, float* y, int32_t T, int64_t n, float decay, int32_t reverse,
                        void* stream) {
  if ((T > 0 && n > 0) && (!x || !y)) { set_error("null tensor"); return SNC_B200_EINVAL; }
  if (T < 0 || n < 0) { set_error("negative size"); return SNC_B200_EINVAL; }
  if (T == 0 || n == 0) return SNC_B200_OK;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // four columns a thread where rows are 16-byte aligned and enough threads
  // remain to fill the device
  const bool quad = n % 4 == 0 && n >= (long long)sms * 1024 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  const long long cols = quad ? n / 4 : n;
  const int grid = (int)std::max(1ll, std::min<long long>((cols + 127) / 128, (long long)sms * 16));
  if (quad) k_leaky_scan<4><<<grid, 128, 0, st>>>(x, y, T, n, decay, reverse ? 1 : 0);
  else k_leaky_scan<1><<<grid, 128, 0, st>>>(x, y, T, n, decay, reverse ? 1 : 0);
  SNCB_CUDA(cudaGetLastError());
  return SNC_B200_OK;
}

int snc_b200_transpose(const float* in, float* out, int32_t T, int32_t I, int32_t J, int64_t st_t,
                       int64_t st_j, void* stream) {
  if (T < 0 || I < 0 || J < 0 || T > 65535) { set_error("transpose: bad size"); return SNC_B200_EINVAL; }
  if ((long long)T * I * J == 0) return SNC_B200_OK;
  if (!in || !out) { set_error("transpose: null tensor"); return SNC_B200_EINVAL; }
  if ((J + 31) / 32 > 65535) { set_error("transpose: J too large"); return SNC_B200_EINVAL; }
  const dim3 grid((unsigned)((I + kTrTile - 1) / kTrTile), (unsigned)((J + kTrTile - 1) / kTrTile), (unsigned)T);
  const bool vi = (reinterpret_cast<uintptr_t>(in) & 15) == 0 && st_t % 4 == 0 && st_j % 4 == 0;
  const bool vo = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && J % 4 == 0;
  auto kern = vi ? (vo ? k_transpose_tile<true, true> : k_transpose_tile<true, false>)
                 : (vo ? k_transpose_tile<false, true> : k_transpose_tile<false, false>);
  kern<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(in, out, I, J, st_t, st_j);
  SNCB_CUDA(cudaGetLastError());
  return SNC_B200_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Forward without device allocation.
//
// Some callers cannot allocate device memory at the moment they run the
// forward: a framework whose caching allocator owns all of the device's memory
// (an allocation behind its back can fail or push it out of memory), and a
// real-time loop that must not pay cudaMalloc's latency or risk its failure in
// the middle of a run.  snc_b200_bptt_forward may allocate on its first use at
// a given size (the per-neuron state buffer of the handle grows on demand).
// This variant runs the same kernel with its scratch -- the membrane
// potential of every (neuron, sample) and the barrier / error words -- in one
// fixed array in device memory that the library reserves statically, so the
// call itself never allocates.  Like the regular forward it ends by reading
// the kernel's error word back and waiting for `stream`.
// ---------------------------------------------------------------------------
namespace sncb {

constexpr size_t kStaticScratchBytes = size_t(4) << 20;  // 4 MiB per device
constexpr size_t kStaticCtlBytes = 256;                   // barrier counter + error word

// Every device that loads the library holds this array until the process exits.
static __device__ __align__(256) unsigned char g_bptt_static_scratch[kStaticScratchBytes];

static std::mutex g_static_mu;
static void* g_static_addr[64] = {};

// Device address of the static scratch on the current device.  The host-side
// symbol is only a stand-in for the array, not a device address, so it is
// looked up once per device (with that device current) and cached.
static int static_scratch(void** out) {
  int dev = 0;
  SNCB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("static scratch: device ordinal beyond 63");
    return SNC_B200_EUNSUPPORTED;
  }
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (!g_static_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_bptt_static_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_bptt_static_scratch)");
    g_static_addr[dev] = p;
  }
  *out = g_static_addr[dev];
  return SNC_B200_OK;
}

}  // namespace sncb

extern "C" int snc_b200_bptt_forward_static(snc_b200_bptt* h, const float* w, const float* ext,
                                            int32_t T, int32_t B, float threshold, float decay,
                                            float slope, int32_t ckpt_every, int32_t smooth,
                                            float* spikes, uint32_t* spike_bits, float* v_saved,
                                            void* stream) {
  using namespace sncb;
  if (!h || !w || !ext || !spikes || !v_saved || T < 1 || B < 1 || ckpt_every < 0 ||
      (!smooth && !spike_bits)) {
    set_error("bptt_forward_static: bad argument");
    return SNC_B200_EINVAL;
  }
  const size_t need = (size_t)h->N * (size_t)B * sizeof(float);
  if (need > kStaticScratchBytes - kStaticCtlBytes) {
    set_error("bptt_forward_static: num_neurons x batch = " + std::to_string((size_t)h->N * B) +
              " exceeds the static scratch limit of " +
              std::to_string((kStaticScratchBytes - kStaticCtlBytes) / sizeof(float)) +
              " (use snc_b200_bptt_forward)");
    return SNC_B200_EUNSUPPORTED;
  }
  void* base = nullptr;
  int rc = static_scratch(&base);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned* ctl = static_cast<unsigned*>(base);
  int* err = reinterpret_cast<int*>(static_cast<char*>(base) + 16);
  float* v = reinterpret_cast<float*>(static_cast<char*>(base) + kStaticCtlBytes);
  // the same launch as snc_b200_bptt_forward (resident when the handle's
  // degrees allow it; a resident launch needs shared memory only)
  BpArgs a = forward_args(h, w, ext, T, B, threshold, decay, slope, ckpt_every, smooth, spikes,
                          spike_bits, v_saved);
  a.v = v;  // zeroed by the kernel before the first step
  a.ctl = ctl;
  a.err = err;
  // the previous call's barrier count and error word must not leak into this one
  SNCB_CUDA(cudaMemsetAsync(base, 0, kStaticCtlBytes, st));
  if ((rc = launch(true, smooth != 0, a, h->sm_count, st))) return rc;
  int e = 0;
  SNCB_CUDA(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  SNCB_CUDA(cudaStreamSynchronize(st));
  if (e) {
    set_error("bptt_forward_static: device barrier timed out");
    return e;
  }
  return SNC_B200_OK;
}
