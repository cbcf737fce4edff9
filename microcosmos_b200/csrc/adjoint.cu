// Reverse-mode derivative of a rollout (the gradient path behind the autograd bindings).
//
// A gradient plan wraps one forward plan (the same kernels as mc_rollout) and adds:
//   * checkpoints of the state every S steps during the forward rollout (S ~ sqrt(T));
//   * per segment, a recompute of its S step inputs with the forward plan;
//   * per step, in reverse, a "tape" recompute of the step's intermediates (steric-corrected
//     prediction, the PBD iterates, the IB stencils and multi-direct forcing iterates) and
//     the adjoint kernels of stream+collide, IB, PBD and steric.
//
// Derivative conventions are those jax.grad applies to the reference: the Peskin stencil
// positions are stop_gradient-ed (src/microcosmos/solver/fluid.py:237-239), floor has
// derivative 0, mod derivative 1, max/min pass the cotangent to the selected argument and
// split it on ties.  Every scatter-add of the adjoint (IB spread, node reaction, steric
// sample weights) goes through a cell-sorted list (CSR) whose entries are ordered by their
// flat index, so sums are taken in a fixed order and gradients are reproducible bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/microcosmos_b200.h"
#include "lbm_cell.cuh"
#include "mc_internal.cuh"

namespace mc {
// Inside a rollout of a one-rollout plan: the current populations in fields.f_grid layout
// written to dst, the rollout left as it is (runtime.cu).
mc_status rollout_snapshot_f(mc_plan* p, float* dst, cudaStream_t s);
}  // namespace mc

namespace {

constexpr int kMaxKK = 64;       // stencil entries per node (kernel size <= 8)
// IB points per CTA of the forcing rounds: bound by the load latency of a point's 16 gathers, so a
// few hundred points go over a dozen SMs and not over two (384 points: interpolation 5.6 -> 3.7 us,
// node side of the reverse 6.3 -> 3.3 us against 256 threads)
constexpr int kPointThreads = 32;
constexpr int kCellBucket = 16;  // entries of a cell ordered in registers
constexpr long long kMaxCells = 4096LL * 4096;  // largest grid of the gradient path
constexpr size_t kOverlapBytes = size_t(1) << 30;  // of a segment's inputs, up to which they are kept twice
constexpr int kDirectSteps = 64;    // steps up to which a plan's first gradient launches forward steps without
                                    // graphs (step_graphs)
constexpr int kDirectReverse = 16;  // the same for reverse steps
constexpr int kPbdThreads = 256;  // threads per rod component in the PBD kernels
constexpr int kPbdRod = 128;      // edges, nodes and pairs of a component kept one per thread

// Per-step inputs of one reverse step, read on the device so that the same CUDA graph
// replays every step of a segment (sa[*jp], jp counts down).
struct StepArgs {
  int t;
  const float* pos;
  const float* vel;
  const float* th;
  const float* f;
  const float* V;
  float* lf_in;
  float* lf_out;
};

struct AD {
  int H, W, N, E, B, HW, C, iters, K, KK, steric, fluid, nskip, has_act;
  int lH, lW, lHW;  // the fluid lattice (f_grid (9, lH, lW)); H, W, HW: the domain grid
  int solver;  // MC_SOLVER_PBD or MC_SOLVER_COSSERAT
  int force_clamp;  // enable_force_clamp: F = F_raw * clamp factor of F_raw
  int NI;      // IB points: N, or 2N with synthetic pairs (point p < N: node p, + side; else node p - N, - side)
  float syn_w, syn_ms;  // synthetic_node_width and the mean lattice scale it is multiplied by
  float dt, damp, st_strength, sigma, scatter, kstretch, kshear, vmax, relax, mass, wp, wm, cp, cm;
  float cos_w;  // stable-Cosserat inertia weight 1 / solver_dt^2
  float scx, scy, sdtx, sdty;
  // topology
  const int2* pairs;
  const int2* bpairs;
  const int* n_start;  // node -> incident edges: entry = e * 2 + role (0: src, 1: tgt)
  const int* n_list;
  const int* e_start;  // edge -> incident bending pairs: entry = b * 2 + role (0: e_in, 1: e_out)
  const int* e_list;
  // rod components (connected by edges): their nodes, edges and bending pairs, ascending
  int ncomp;
  const int* c_nstart;
  const int* c_nodes;
  const int* c_estart;
  const int* c_edges;
  const int* c_bstart;
  const int* c_bps;
  // per-step inputs of the reverse step being replayed
  const StepArgs* sa;
  int* jp;
  const float* ndeg;
  const float* edeg;
  const float* rest_len;
  const float* kb;
  const float* rest_static;
  const float* act_c;
  const float* act_amp;
  const float* act_om;
  const float* act_ph;
  // tape
  float* rest;   // (B) rest angles of the current step
  float2* pred0;  // (N)
  float2* pp;     // (C+1) x N PBD iterates
  float* tt;      // (C+1) x E
  int* ib_idx;    // NI x KK
  float* ib_w;    // NI x KK
  float2* sraw;   // iters x NI
  float2* s_tmp;  // NI
  float2* uc;     // lHW
  float* inv;     // lHW
  // entries (stencil entries of the IB points, or steric samples) by cell: a cell's entries are
  // collected in its bucket (beyond kCellBucket in its overflow list) as they arrive, then ordered
  // into its run of ent; used for the lattice, then for the domain grid
  int* cnt;       // max(HW, lHW): entries of the cell, zero between uses
  int* bucket;    // max(HW, lHW) x kCellBucket
  int* ovf_head;  // max(HW, lHW): first overflow entry of the cell, -1 between uses
  int* ovf_next;
  int* ovf;
  int* start;     // max(HW, lHW): run of a cell with entries
  int* ent;       // runs: kCellBucket per touched cell, longer ones in the pool behind
  int pool;       // where the pool begins
  int* touched;   // cells with at least one entry (any order)
  int* ntouched;  // [0] their count, [1] overflow entries, [2] use of the pool
  // adjoint
  float* lf0p;   // 9 x lHW
  float* lv;     // 2 x lHW
  float* lrho;   // lHW
  float2* luc;   // lHW
  float2* lnv;   // NI
  float2* lprev;  // N
  float2* lpos;   // N   (state cotangent)
  float2* lvel;   // N
  float* lth;     // E
  float2* lp[2];  // N
  float* lt[2];   // E
  float2* lcur;   // E
  float* lthn;    // E
  float* gb;      // B
  float2* ly;     // N  stable-Cosserat: cotangent of the prediction the iterations pull toward
  float2* lfn;    // N  stable-Cosserat: cotangent of a node's summed force
  float* lhn;     // N  stable-Cosserat: cotangent of a node's summed stiffness
  float* rest_acc;  // B (this step)
  float* d_c;
  float* d_amp;
  float* d_ph;
  float* d_om;
  float* d_rest;
  float* d_len;
  float* d_kb;
  // steric
  float* st_val;   // 16 N
  float2* lpred1;  // N
  float2* lpred0p;  // N
  float* lV;       // HW
  float* ctmp;     // HW
  float* ldep;     // HW
};

__device__ __forceinline__ float dmaxf(float x, float c) { return x > c ? 1.0f : (x == c ? 0.5f : 0.0f); }

// cotangent of (x, y) through (x c, y c), c = min(1, vmax / (sqrt(x^2+y^2+eps)+eps))
__device__ __forceinline__ float2 clamp_vjp(float x, float y, float vmax, float gx, float gy) {
  const float mag = sqrtf((x * x + y * y) + MC_EPSIL);
  const float a = vmax / (mag + MC_EPSIL);
  const float c = mc::min_prop(1.0f, a);
  const float sel = a < 1.0f ? 1.0f : (a == 1.0f ? 0.5f : 0.0f);
  const float gc = x * gx + y * gy;
  const float da = -vmax / ((mag + MC_EPSIL) * (mag + MC_EPSIL));
  const float k = ((gc * sel) * da) / mag;
  return make_float2(c * gx + k * x, c * gy + k * y);
}

__device__ __forceinline__ int cell_of(int y, int x, int H, int W) { return mc::imod_floor(y, H) * W + mc::imod_floor(x, W); }

// map_coordinates(order=1, mode="wrap") of field V at (yy, xx)
__device__ __forceinline__ float sample_wrap(const float* V, int H, int W, float yy, float xx) {
  const float ly = floorf(yy), lx = floorf(xx);
  const float ty = yy - ly, tx = xx - lx;
  const float wy0 = 1.0f - ty, wx0 = 1.0f - tx;
  const int iy = (int)ly, ix = (int)lx;
  const int y0 = mc::imod_floor(iy, H), y1 = mc::imod_floor(iy + 1, H);
  const int x0 = mc::imod_floor(ix, W), x1 = mc::imod_floor(ix + 1, W);
  float acc = (wy0 * wx0) * V[y0 * W + x0];
  acc = acc + (wy0 * tx) * V[y0 * W + x1];
  acc = acc + (ty * wx0) * V[y1 * W + x0];
  acc = acc + (ty * tx) * V[y1 * W + x1];
  return acc;
}

// ------------------------------------------------------------------ tape: prediction + steric
__global__ void k_rest(AD d) {
  mc::after_previous();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= d.B) return;
  const int t = d.sa[*d.jp].t;
  float r;
  if (d.has_act) {
    const float arg = d.act_om[b] * (float)t + d.act_ph[b];
    r = d.act_c[b] + d.act_amp[b] * sinf(arg);
  } else {
    r = d.rest_static[b];
  }
  d.rest[b] = r;
  d.rest_acc[b] = 0.0f;
}

// 4 lanes per node, as the forward node-step kernel: one finite-difference sample and a quarter of
// the neighbours each, their terms added in neighbour order.  384 nodes: 8.6 -> 4.1 us against one
// thread per node.
__global__ void __launch_bounds__(128) k_pred(AD d) {
  mc::after_previous();
  const StepArgs a = d.sa[*d.jp];
  const float2* __restrict__ pos = reinterpret_cast<const float2*>(a.pos);
  const float2* __restrict__ vel = reinterpret_cast<const float2*>(a.vel);
  const float* __restrict__ theta = a.th;
  const float* __restrict__ V = a.V;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < d.E) d.tt[t] = theta[t];
  const int i = min(t >> 2, d.N - 1), qs = t & 3;
  const bool on = (t >> 2) < d.N;
  const unsigned full = 0xffffffffu;
  const float2 p = pos[i], v = vel[i];
  float2 q = make_float2(p.x + (v.x * d.damp) * d.dt, p.y + (v.y * d.damp) * d.dt);
  if (on && qs == 0) d.pred0[i] = q;
  if (d.steric) {
    const float Wf = (float)d.W, Hf = (float)d.H;
    const float x = mc::fmod_floor(q.x, Wf), y = mc::fmod_floor(q.y, Hf);
    const float e = (qs & 1) ? -0.5f : 0.5f, den = 1.0f;
    const float s = sample_wrap(V, d.H, d.W, qs < 2 ? y : y + e, qs < 2 ? x + e : x);
    const float xp = __shfl_sync(full, s, 0, 4), xm = __shfl_sync(full, s, 1, 4);
    const float yp = __shfl_sync(full, s, 2, 4), ym = __shfl_sync(full, s, 3, 4);
    float fx = -((xp - xm) / den), fy = -((yp - ym) / den);
    if (d.nskip > 0) {
      const float inv2s2 = 2.0f * d.sigma * d.sigma;
      const float norm = (float)(2.0 * M_PI) * d.sigma * d.sigma;
      float ax = 0.0f, ay = 0.0f;
      // the neighbours' wrapped predictions, recomputed from their positions and velocities
      for (int o0 = -d.nskip; o0 <= d.nskip; o0 += 4) {
        const int o = o0 + qs, j = i + o;
        float tx = 0.0f, ty = 0.0f;
        if (o <= d.nskip && o != 0 && j >= 0 && j < d.N) {  // a node's own term is zero
          const float2 pj0 = pos[j], vj = vel[j];
          const float qx = pj0.x + (vj.x * d.damp) * d.dt, qy = pj0.y + (vj.y * d.damp) * d.dt;
          const float2 r = mc::min_image(x, y, mc::fmod_floor(qx, Wf), mc::fmod_floor(qy, Hf), Wf, Hf);
          const float d2 = r.x * r.x + r.y * r.y;
          const float K = expf(-d2 / inv2s2) / norm;
          tx = K * r.x;
          ty = K * r.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          ax = ax + __shfl_sync(full, tx, k, 4);
          ay = ay + __shfl_sync(full, ty, k, 4);
        }
      }
      const float pre = d.scatter / (d.sigma * d.sigma);
      fx = fx - pre * ax;
      fy = fy - pre * ay;
    }
    q.x = q.x + (fx * d.st_strength) * d.dt;
    q.y = q.y + (fy * d.st_strength) * d.dt;
  }
  if (on && qs == 0) d.pp[i] = q;
}

// ------------------------------------------------------------------ tape: PBD iterates (one CTA)
// bending correction of pair (e_in, e_out) from the angles th_in = theta[e_in], th_out = theta[e_out]
__device__ __forceinline__ float bend_corr_v(float th_in, float th_out, float rest, float kb) {
  const float pi = (float)M_PI;
  const float diff = mc::fmod_floor((th_out - th_in) + pi, (float)(2.0 * M_PI)) - pi;
  return ((diff - rest) * kb) * 0.5f;
}

__device__ __forceinline__ float bend_corr(const AD& d, const float* th, int b) {
  const int2 bp = d.bpairs[b];
  return bend_corr_v(th[bp.x], th[bp.y], d.rest[b], d.kb[b]);
}

// stretch + shear force of an edge from its endpoints a = p[src], b = p[tgt], its new angle
// and its rest length
__device__ __forceinline__ float2 edge_force_v(const AD& d, float2 a, float2 b, float thn, float L0) {
  const float tx = cosf(thn) * L0, ty = sinf(thn) * L0;
  const float2 cur = mc::min_image(b.x, b.y, a.x, a.y, (float)d.W, (float)d.H);
  const float L = sqrtf(cur.x * cur.x + cur.y * cur.y);
  const float m = mc::max_prop(L, 1e-8f);
  const float sx = (cur.x / m) * (L - L0), sy = (cur.y / m) * (L - L0);
  const float shx = (cur.x - tx) - sx, shy = (cur.y - ty) - sy;
  return make_float2(((sx + shx * d.kshear) * d.kstretch) * 0.5f, ((sy + shy * d.kshear) * d.kstretch) * 0.5f);
}

__device__ __forceinline__ float2 edge_force(const AD& d, const float2* p, float thn, int e) {
  const int2 pr = d.pairs[e];
  return edge_force_v(d, p[pr.x], p[pr.y], thn, d.rest_len[e]);
}

// Rod components whose edges, nodes and bending pairs fit one per thread, with at most
// kPbdGather incidences each (chains: 2), keep their topology in registers and what the threads
// exchange in shared memory for all C iterations; the tape in global memory is written but not
// read back.  As in the forward rod kernel (rod.cuh) the angle passes, which read no position, run
// first; the sines, cosines and (in the reverse pass) everything else that depends on the tape
// alone is computed for all iterations at once, by all threads; the recurrences that remain are a
// few operations per iteration.  Same operands and summation order as the general loops below, so
// the same bits.  Measured (256^2, 8 x 48 nodes, one launch alone with warm caches): tape 36.6 -> 22.8 us,
// reverse 38.4 -> 28.6 us; before, each phase of an iteration went through the tape in global memory.
constexpr int kPbdGather = 4;
constexpr int kTapeChunk = 20;  // iterations whose angles and rest vectors the tape kernel keeps at a time
constexpr int kRevChunk = 10;   // iterations whose tables the reverse kernel keeps at a time

// v / n for a degree n; r = 1 / n is exact for 1, 2 and 4
__device__ __forceinline__ float div_degree(float v, float n, float r) {
  return n == 1.0f || n == 2.0f || n == 4.0f ? v * r : v / n;
}

// place of g in the ascending list[a..b); -1 when it is not a member
__device__ __forceinline__ int local_of(const int* __restrict__ list, int a, int b, int g) {
  const int first = list[a], last = list[b - 1];
  if (g < first || g > last) return -1;
  if (last - first == b - 1 - a) return g - first;
  int lo = a, hi = b - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (list[mid] < g) lo = mid + 1; else hi = mid;
  }
  return list[lo] == g ? lo - a : -1;
}

struct PbdEdgeReg {  // an edge and its bending pairs (edge pass of the forward)
  int e = -1, nb = 0;
  int2 bp[kPbdGather];
  float rest[kPbdGather], kb[kPbdGather];
  bool neg[kPbdGather];
  float edeg = 1.0f;
};

struct PbdNodeReg {  // a node and its incident edges
  int n = -1, ne = 0;
  int e[kPbdGather];
  int2 pr[kPbdGather];
  float L0[kPbdGather];
  bool neg[kPbdGather];
  float ndeg = 1.0f;
};

// loads thread t's edge / node of component c; false when a list is too long for registers
__device__ __forceinline__ bool pbd_load_edge(const AD& d, int ie, int eb, PbdEdgeReg& r) {
  if (ie >= eb) return true;
  r.e = d.c_edges[ie];
  const int qa = d.e_start[r.e], qb = d.e_start[r.e + 1];
  r.nb = qb - qa;
  if (r.nb > kPbdGather) return false;
#pragma unroll
  for (int q = 0; q < kPbdGather; ++q)
    if (q < r.nb) {
      const int en = d.e_list[qa + q];
      r.bp[q] = d.bpairs[en >> 1];
      r.rest[q] = d.rest[en >> 1];
      r.kb[q] = d.kb[en >> 1];
      r.neg[q] = en & 1;
    }
  r.edeg = d.edeg[r.e];
  return true;
}

__device__ __forceinline__ bool pbd_load_node(const AD& d, int in, int nb, PbdNodeReg& r) {
  if (in >= nb) return true;
  r.n = d.c_nodes[in];
  const int qa = d.n_start[r.n], qb = d.n_start[r.n + 1];
  r.ne = qb - qa;
  if (r.ne > kPbdGather) return false;
#pragma unroll
  for (int q = 0; q < kPbdGather; ++q)
    if (q < r.ne) {
      const int en = d.n_list[qa + q];
      r.e[q] = en >> 1;
      r.pr[q] = d.pairs[en >> 1];
      r.L0[q] = d.rest_len[en >> 1];
      r.neg[q] = en & 1;
    }
  r.ndeg = d.ndeg[r.n];
  return true;
}

// The tape of a component that fits; false (nothing done) when it does not.
__device__ __forceinline__ bool pbd_fwd_fast(const AD& d, int ea, int eb, int na, int nb) {
  __shared__ float ths[kTapeChunk + 1][kPbdRod];  // row k: the angles before pass k of the chunk
  __shared__ float2 vec[kTapeChunk][kPbdRod];     // rest vectors after pass k
  __shared__ float2 ps[kPbdRod], fs[kPbdRod];
  __shared__ float l0s[kPbdRod];
  const int tid = threadIdx.x, ne = eb - ea;
  PbdEdgeReg re;
  PbdNodeReg rn;
  bool ok = ne <= kPbdRod && nb - na <= kPbdRod;
  if (ok) ok = pbd_load_edge(d, ea + tid, eb, re) && pbd_load_node(d, na + tid, nb, rn);
  // places in the component instead of global indices
  int2 ends = make_int2(0, 0);
  if (ok && re.e >= 0) {
    const int2 pr = d.pairs[re.e];
    ends = make_int2(local_of(d.c_nodes, na, nb, pr.x), local_of(d.c_nodes, na, nb, pr.y));
#pragma unroll
    for (int q = 0; q < kPbdGather; ++q)
      if (q < re.nb) {
        re.bp[q] = make_int2(local_of(d.c_edges, ea, eb, re.bp[q].x), local_of(d.c_edges, ea, eb, re.bp[q].y));
        if (re.bp[q].x < 0 || re.bp[q].y < 0) ok = false;
      }
  }
  if (!__syncthreads_and(ok)) return false;
  const float er = 1.0f / re.edeg, nr = 1.0f / rn.ndeg;
  if (re.e >= 0) {
    l0s[tid] = d.rest_len[re.e];
    ths[0][tid] = d.tt[re.e];
  }
  if (rn.n >= 0) {
#pragma unroll
    for (int q = 0; q < kPbdGather; ++q)
      if (q < rn.ne) rn.e[q] = local_of(d.c_edges, ea, eb, rn.e[q]);
    ps[tid] = d.pp[rn.n];
  }
  __syncthreads();
  const float ksh = d.kshear, kst = d.kstretch, Wf = (float)d.W, Hf = (float)d.H;
  for (int k0 = 0; k0 < d.C; k0 += kTapeChunk) {
    const int q = min(kTapeChunk, d.C - k0);
    for (int k = 0; k < q; ++k) {
      if (re.e >= 0) {
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < kPbdGather; ++i)
          if (i < re.nb) {
            const float cr = bend_corr_v(ths[k][re.bp[i].x], ths[k][re.bp[i].y], re.rest[i], re.kb[i]);
            acc = acc + (re.neg[i] ? -cr : cr);
          }
        const float t = ths[k][tid] + div_degree(acc, re.edeg, er) * 1.8f;
        ths[k + 1][tid] = t;
        d.tt[(size_t)(k0 + k + 1) * d.E + re.e] = t;
      }
      __syncthreads();
    }
    for (int k = tid >> 5; k < q; k += kPbdThreads / 32)
      for (int e = tid & 31; e < ne; e += 32) {
        const float t = ths[k + 1][e];
        vec[k][e] = make_float2(cosf(t) * l0s[e], sinf(t) * l0s[e]);
      }
    __syncthreads();
    if (re.e >= 0) ths[0][tid] = ths[q][tid];
    for (int k = 0; k < q; ++k) {
      if (re.e >= 0) {
        const float2 a = ps[ends.x], b = ps[ends.y], tv = vec[k][tid];
        const float L0 = l0s[tid];
        const float2 cur = mc::min_image(b.x, b.y, a.x, a.y, Wf, Hf);
        const float L = sqrtf(cur.x * cur.x + cur.y * cur.y);
        const float m = mc::max_prop(L, 1e-8f);
        const float sx = (cur.x / m) * (L - L0), sy = (cur.y / m) * (L - L0);
        const float shx = (cur.x - tv.x) - sx, shy = (cur.y - tv.y) - sy;
        fs[tid] = make_float2(((sx + shx * ksh) * kst) * 0.5f, ((sy + shy * ksh) * kst) * 0.5f);
      }
      __syncthreads();
      if (rn.n >= 0) {
        float ax = 0.0f, ay = 0.0f;
#pragma unroll
        for (int i = 0; i < kPbdGather; ++i)
          if (i < rn.ne) {
            const float2 f = fs[rn.e[i]];
            if (rn.neg[i]) {
              ax = ax + (-f.x);
              ay = ay + (-f.y);
            } else {
              ax = ax + f.x;
              ay = ay + f.y;
            }
          }
        const float2 self = ps[tid];
        const float2 moved =
            make_float2(self.x + div_degree(ax, rn.ndeg, nr), self.y + div_degree(ay, rn.ndeg, nr));
        ps[tid] = moved;
        d.pp[(size_t)(k0 + k + 1) * d.N + rn.n] = moved;
      }
      __syncthreads();
    }
  }
  return true;
}

// one CTA per rod component: the components never interact in the PBD passes
__global__ void __launch_bounds__(kPbdThreads, 2) k_pbd_fwd(AD d) {
  mc::after_previous();
  const int c = blockIdx.x;
  const int ea = d.c_estart[c], eb = d.c_estart[c + 1], na = d.c_nstart[c], nb = d.c_nstart[c + 1];
  if (pbd_fwd_fast(d, ea, eb, na, nb)) return;
  for (int k = 0; k < d.C; ++k) {
    const float* th = d.tt + (size_t)k * d.E;
    float* thn = d.tt + (size_t)(k + 1) * d.E;
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      float acc = 0.0f;
      for (int q = d.e_start[e]; q < d.e_start[e + 1]; ++q) {
        const int en = d.e_list[q];
        const float c = bend_corr(d, th, en >> 1);
        acc = acc + ((en & 1) ? -c : c);
      }
      thn[e] = th[e] + (acc / d.edeg[e]) * 1.8f;
    }
    __syncthreads();
    const float2* p = d.pp + (size_t)k * d.N;
    float2* pn = d.pp + (size_t)(k + 1) * d.N;
    for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
      const int n = d.c_nodes[in];
      float ax = 0.0f, ay = 0.0f;
      for (int q = d.n_start[n]; q < d.n_start[n + 1]; ++q) {
        const int en = d.n_list[q];
        const int e = en >> 1;
        const float2 f = edge_force(d, p, thn[e], e);
        if (en & 1) {
          ax = ax + (-f.x);
          ay = ay + (-f.y);
        } else {
          ax = ax + f.x;
          ay = ay + f.y;
        }
      }
      const float dg = d.ndeg[n];
      pn[n] = make_float2(p[n].x + ax / dg, p[n].y + ay / dg);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ entries by cell
__device__ __forceinline__ void cell_append(const AD& d, int cell, int e) {
  const int pos = atomicAdd(d.cnt + cell, 1);
  if (pos == 0) d.touched[atomicAdd(d.ntouched, 1)] = cell;
  if (pos < kCellBucket) {
    d.bucket[(size_t)cell * kCellBucket + pos] = e;
  } else {
    const int o = atomicAdd(d.ntouched + 1, 1);
    d.ovf[o] = e;
    d.ovf_next[o] = atomicExch(d.ovf_head + cell, o);
  }
}

// Sorts R keys in registers.
template <int R>
__device__ __forceinline__ void sort_keys(int (&k)[R]) {
#pragma unroll
  for (int size = 2; size <= R; size <<= 1)
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int o = i ^ j;
        if (o > i) {
          const int lo = min(k[i], k[o]), hi = max(k[i], k[o]);
          k[i] = (i & size) == 0 ? lo : hi;
          k[o] = (i & size) == 0 ? hi : lo;
        }
      }
}

template <int R>
__device__ __forceinline__ void order_row(const AD& d, int i, int cell, int len) {
  int k[R];
  const int4* bucket = reinterpret_cast<const int4*>(d.bucket + (size_t)cell * kCellBucket);
  int4* row = reinterpret_cast<int4*>(d.ent + (size_t)i * kCellBucket);
#pragma unroll
  for (int q = 0; q < R; q += 4) {
    int4 v = make_int4(0, 0, 0, 0);
    if (q < len) v = bucket[q / 4];
    k[q] = q < len ? v.x : 0x7fffffff;
    k[q + 1] = q + 1 < len ? v.y : 0x7fffffff;
    k[q + 2] = q + 2 < len ? v.z : 0x7fffffff;
    k[q + 3] = q + 3 < len ? v.w : 0x7fffffff;
  }
  sort_keys<R>(k);
#pragma unroll
  for (int q = 0; q < R; q += 4)
    if (q < len) row[q / 4] = make_int4(k[q], k[q + 1], k[q + 2], k[q + 3]);
}

// The entries of each touched cell in increasing index (the order np.add.at applies them): one
// thread per cell sorts up to 16 in registers, its warp ranks longer ones.  Replaces a count, three
// scans over all cells, a fill, a compaction and an insertion sort in global memory (24 to 31 us at
// 256^2) by this launch of 3.6 us.
__global__ void __launch_bounds__(128) k_cell_order(AD d) {
  mc::after_previous();
  const int n = *d.ntouched;
  const int i0 = blockIdx.x * blockDim.x;
  if (i0 >= n) return;
  const int i = i0 + threadIdx.x, lane = threadIdx.x & 31;
  const bool on = i < n;
  const int cell = on ? d.touched[i] : 0;
  const int len = on ? d.cnt[cell] : 0;
  if (len > 0 && len <= 8) order_row<8>(d, i, cell, len);
  if (len > 8 && len <= kCellBucket) order_row<kCellBucket>(d, i, cell, len);
  if (len > 0 && len <= kCellBucket) d.start[cell] = i * kCellBucket;
  for (unsigned deep = __ballot_sync(0xffffffffu, len > kCellBucket); deep; deep &= deep - 1) {
    const int src = __ffs(deep) - 1;
    const int c = __shfl_sync(0xffffffffu, cell, src), m = __shfl_sync(0xffffffffu, len, src);
    int base = 0;
    if (lane == 0) base = atomicAdd(d.ntouched + 2, 2 * m);
    int* raw = d.ent + d.pool + __shfl_sync(0xffffffffu, base, 0);
    int* run = raw + m;
    const int* bucket = d.bucket + (size_t)c * kCellBucket;
    if (lane < kCellBucket) raw[lane] = bucket[lane];
    if (lane == 0) {
      int e = d.ovf_head[c];
      for (int q = kCellBucket; q < m; ++q) {
        raw[q] = d.ovf[e];
        e = d.ovf_next[e];
      }
      d.ovf_head[c] = -1;
      d.start[c] = (int)(run - d.ent);
    }
    __syncwarp();
    for (int q = lane; q < m; q += 32) {
      const int k = raw[q];
      int rank = 0;
      for (int o = 0; o < m; ++o) rank += raw[o] < k ? 1 : 0;
      run[rank] = k;
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------ tape: IB stencils
// The stencil of IB point n at the step's final PBD positions; with synthetic pairs the
// point is offset by +-syn_w * syn_ms along the normal of its node's chain tangent (the sum
// of its edges' min-image vectors, src roles first, as the forward computes it).  The
// positions are stop_gradient-ed: constants of the derivative.
__device__ __forceinline__ float2 tape_point(const AD& d, int n) {
  const int gi = n < d.N ? n : n - d.N;
  const float2* pc = d.pp + (size_t)d.C * d.N;
  const float2 p = pc[gi];
  float x = p.x * d.scx, y = p.y * d.scy;
  if (d.NI > d.N) {
    float tx = 0.0f, ty = 0.0f;
    for (int q = d.n_start[gi]; q < d.n_start[gi + 1]; ++q) {
      const int2 pr = d.pairs[d.n_list[q] >> 1];
      const float2 ev = mc::min_image(pc[pr.y].x, pc[pr.y].y, pc[pr.x].x, pc[pr.x].y, (float)d.W, (float)d.H);
      tx = tx + ev.x;
      ty = ty + ev.y;
    }
    const float nrm = sqrtf((tx * tx + ty * ty) + MC_EPSIL);
    const float ux = tx / nrm, uy = ty / nrm;
    const float ox = (d.syn_w * (-uy)) * d.syn_ms, oy = (d.syn_w * ux) * d.syn_ms;
    if (n < d.N) {
      x = x + ox;
      y = y + oy;
    } else {
      x = x - ox;
      y = y - oy;
    }
  }
  return make_float2(x, y);
}

// any kernel size, one thread per IB point
__global__ void k_ib_weights(AD d) {
  mc::after_previous();
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= d.NI) return;
  const float2 g = tape_point(d, n);
  const float x = g.x, y = g.y;
  const int K = d.K;
  const float half = (float)((K - 1) / 2);
  const float hw = (float)K / 2.0f;
  const float sx = floorf(x) - half, sy = floorf(y) - half;
  float w[kMaxKK];
  float s = 0.0f;
  for (int a = 0; a < K; ++a) {
    for (int b = 0; b < K; ++b) {
      const float nx = sx + (float)a, ny = sy + (float)b;
      const float rx = fabsf(nx - x) / hw, ry = fabsf(ny - y) / hw;
      const float px = rx <= 2.0f ? 0.25f * (1.0f + cosf(((float)M_PI * rx) / 2.0f)) : 0.0f;
      const float py = ry <= 2.0f ? 0.25f * (1.0f + cosf(((float)M_PI * ry) / 2.0f)) : 0.0f;
      const int q = a * K + b;
      w[q] = px * py;
      s = s + w[q];
      const int cell = cell_of((int)ny, (int)nx, d.lH, d.lW);
      d.ib_idx[(size_t)n * d.KK + q] = cell;
      cell_append(d, cell, n * d.KK + q);
    }
  }
  for (int q = 0; q < d.KK; ++q) d.ib_w[(size_t)n * d.KK + q] = w[q] / (s + MC_EPSIL);
}

// K <= 4: 4 lanes per IB point, lane a a column of the stencil (as k_stencil4 of the forward).
// 384 points: 9.4 -> 5.8 us against one thread per point.
__global__ void __launch_bounds__(128) k_ib_weights4(AD d) {
  mc::after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = min(t >> 2, d.NI - 1), a = t & 3, K = d.K;
  const bool mine = (t >> 2) < d.NI && a < K;
  const float2 g = tape_point(d, n);
  const float half = (float)((K - 1) / 2), hw = (float)K / 2.0f;
  const float nx = (floorf(g.x) - half) + (float)a, ny = (floorf(g.y) - half) + (float)a;
  const float rx = fabsf(nx - g.x) / hw, ry = fabsf(ny - g.y) / hw;
  const float px = rx <= 2.0f ? 0.25f * (1.0f + cosf(((float)M_PI * rx) / 2.0f)) : 0.0f;
  const float py = ry <= 2.0f ? 0.25f * (1.0f + cosf(((float)M_PI * ry) / 2.0f)) : 0.0f;
  const int cx = mc::imod_floor((int)nx, d.lW), cy = mc::imod_floor((int)ny, d.lH) * d.lW;
  const unsigned full = 0xffffffffu;
  float w[4];
  int cell[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    w[b] = px * __shfl_sync(full, py, b, 4);
    cell[b] = __shfl_sync(full, cy, b, 4) + cx;
  }
  float s = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float we = __shfl_sync(full, w[b], e, 4);
      if (e < K && b < K) s = s + we;
    }
  if (!mine) return;
  const int q0 = (n * K + a) * K;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (b < K) {
      d.ib_idx[q0 + b] = cell[b];
      d.ib_w[q0 + b] = w[b] / (s + MC_EPSIL);
      cell_append(d, cell[b], q0 + b);
    }
}

// ------------------------------------------------------------------ tape: macroscopic + IB iterations
__global__ void k_macro(AD d) {
  mc::after_previous();
  const float* __restrict__ f = d.sa[*d.jp].f;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.lHW) return;
  float r = mc::max_prop(f[c], MC_EPSIL);
  float fv[9];
  fv[0] = r;
#pragma unroll
  for (int i = 1; i < 9; ++i) {
    fv[i] = mc::max_prop(f[(size_t)i * d.lHW + c], MC_EPSIL);
    r = r + fv[i];
  }
  const float rho = mc::max_prop(r, 0.1f);
  const float ux = (((((fv[1] - fv[3]) + fv[5]) - fv[6]) - fv[7]) + fv[8]) / rho;
  const float uy = (((((fv[2] - fv[4]) + fv[5]) + fv[6]) - fv[7]) - fv[8]) / rho;
  const float c1 = mc::clamp_factor(ux, uy, d.vmax);
  d.uc[c] = make_float2(ux * c1, uy * c1);
  float cov = 0.0f;
  const int len = d.cnt[c];
  if (len > 0)
    for (int q = d.start[c], end = q + len; q < end; ++q) cov = cov + d.ib_w[d.ent[q]];
  d.inv[c] = 1.0f / mc::max_prop(cov, 1.0f);
}

// Sum of field(cell) * weight over a point's stencil in stencil order (SCALE: the field is first
// multiplied by d.inv); all loads of a point in flight together.  load() reads what the kernel
// before does not write, past the L1, and may come before the wait for it.
template <int KK, bool SCALE>
struct PointTaps {
  int c[KK];
  float w[KK], sc[SCALE ? KK : 1];
  __device__ __forceinline__ void load(const AD& d, int n) {
    const int base = n * KK;
    if constexpr (KK % 4 == 0) {
#pragma unroll
      for (int q = 0; q < KK; q += 4) {
        const int4 i4 = __ldcg(reinterpret_cast<const int4*>(d.ib_idx + base + q));
        const float4 w4 = __ldcg(reinterpret_cast<const float4*>(d.ib_w + base + q));
        c[q] = i4.x; c[q + 1] = i4.y; c[q + 2] = i4.z; c[q + 3] = i4.w;
        w[q] = w4.x; w[q + 1] = w4.y; w[q + 2] = w4.z; w[q + 3] = w4.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < KK; ++q) {
        c[q] = __ldcg(d.ib_idx + base + q);
        w[q] = __ldcg(d.ib_w + base + q);
      }
    }
    if constexpr (SCALE) {
#pragma unroll
      for (int q = 0; q < KK; ++q) sc[q] = __ldcg(d.inv + c[q]);
    }
  }
  __device__ __forceinline__ float2 sum(const AD&, int, const float2* field) const {
    float2 v[KK];
#pragma unroll
    for (int q = 0; q < KK; ++q) {
      v[q] = field[c[q]];
      if constexpr (SCALE) v[q] = make_float2(sc[q] * v[q].x, sc[q] * v[q].y);
    }
    float ix = 0.0f, iy = 0.0f;
#pragma unroll
    for (int q = 0; q < KK; ++q) {
      ix = ix + v[q].x * w[q];
      iy = iy + v[q].y * w[q];
    }
    return make_float2(ix, iy);
  }
};
// any kernel size
template <bool SCALE>
struct PointTaps<0, SCALE> {
  __device__ __forceinline__ void load(const AD&, int) {}
  __device__ __forceinline__ float2 sum(const AD& d, int n, const float2* field) const {
    const int base = n * d.KK;
    float ix = 0.0f, iy = 0.0f;
    for (int q = 0; q < d.KK; ++q) {
      const int c = d.ib_idx[base + q];
      const float w = d.ib_w[base + q];
      float2 v = field[c];
      if (SCALE) v = make_float2(d.inv[c] * v.x, d.inv[c] * v.y);
      ix = ix + v.x * w;
      iy = iy + v.y * w;
    }
    return make_float2(ix, iy);
  }
};

// Sum of point value * weight over a cell's run, in order: 4 entries in flight, the first 4 loaded
// ahead.
struct CellRun {
  int start, len, e[4];
  float w[4];
  __device__ __forceinline__ void chunk(const AD& d, int j) {
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = j + q < len ? __ldcg(d.ent + start + j + q) : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = j + q < len ? __ldcg(d.ib_w + e[q]) : 0.0f;
  }
  __device__ __forceinline__ void load(const AD& d, int c) {
    start = __ldcg(d.start + c);
    len = __ldcg(d.cnt + c);
    chunk(d, 0);
  }
  __device__ __forceinline__ float2 sum(const AD& d, const float2* value) {
    float ax = 0.0f, ay = 0.0f;
    for (int j = 0; j < len; j += 4) {
      if (j > 0) chunk(d, j);
      float2 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q < len) v[q] = value[d.KK == 16 ? e[q] >> 4 : e[q] / d.KK];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q < len) {
          ax = ax + v[q].x * w[q];
          ay = ay + v[q].y * w[q];
        }
    }
    return make_float2(ax, ay);
  }
};

__device__ __forceinline__ const float2* step_positions(const AD& d) {
  return reinterpret_cast<const float2*>(d.sa[*d.jp].pos);
}

// The multi-direct forcing rounds and their reverse, one launch per phase.  (All phases in one
// launch of a cluster of 8 CTAs with its hardware barrier between them took as long, 48 us against
// 51 for five rounds of 384 points, and longer from 4,096 points: a phase is its dependent loads.)
// Each phase reads before the wait what its predecessor does not write.  k_ib_interp comes behind
// k_macro (uc, inv) or k_ib_spread (uc); k_ib_spread behind k_ib_interp (sraw, s_tmp); k_ib_rev_node
// behind k_lbm_adj1 (luc, lv, lrho, lf0p) or k_ib_rev_cell (luc); k_ib_rev_cell behind k_ib_rev_node
// (lnv, s_tmp).
template <int KK>
__device__ __forceinline__ void tape_interp(const AD& d, int n, int it) {
  PointTaps<KK, false> taps;
  float2 pc, p0;
  const bool on = n < d.NI;
  if (on) {
    const int gi = n < d.N ? n : n - d.N;
    taps.load(d, n);
    pc = __ldcg(d.pp + (size_t)d.C * d.N + gi);
    p0 = __ldcg(step_positions(d) + gi);
  }
  mc::after_previous();
  if (!on) return;
  const float2 u = taps.sum(d, n, d.uc);
  const float v1x = (pc.x - p0.x) / d.dt, v1y = (pc.y - p0.y) / d.dt;
  const float nvx = (v1x * d.scx) * d.dt, nvy = (v1y * d.scy) * d.dt;
  const float sx = (nvx - u.x) * d.relax, sy = (nvy - u.y) * d.relax;
  d.sraw[(size_t)it * d.NI + n] = make_float2(sx, sy);
  const float cf = mc::clamp_factor(sx, sy, d.vmax);
  d.s_tmp[n] = make_float2(sx * cf, sy * cf);
}
template <int KK>
__device__ __forceinline__ void rev_node(const AD& d, int n, int it) {
  PointTaps<KK, true> taps;
  float2 r, a = make_float2(0.0f, 0.0f);
  const bool on = n < d.NI;
  if (on) {
    taps.load(d, n);
    r = __ldcg(d.sraw + (size_t)it * d.NI + n);
    if (it < d.iters - 1) a = __ldcg(d.lnv + n);
  }
  mc::after_previous();
  if (!on) return;
  const float2 s = taps.sum(d, n, d.luc);
  const float2 lr = clamp_vjp(r.x, r.y, d.vmax, s.x, s.y);
  a.x += d.relax * lr.x;
  a.y += d.relax * lr.y;
  d.lnv[n] = a;
  d.s_tmp[n] = make_float2(-d.relax * lr.x, -d.relax * lr.y);
}
__global__ void k_ib_interp(AD d, int it) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;  // IB point
  switch (d.KK) {
    case 16: return tape_interp<16>(d, n, it);
    case 9: return tape_interp<9>(d, n, it);
    case 4: return tape_interp<4>(d, n, it);
    default: return tape_interp<0>(d, n, it);
  }
}
__global__ void k_ib_spread(AD d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < __ldcg(d.ntouched);
  CellRun run;
  int c = 0;
  float iv = 0.0f;
  float2 u;
  if (on) {
    c = __ldcg(d.touched + i);
    run.load(d, c);
    iv = __ldcg(d.inv + c);
    u = __ldcg(d.uc + c);
  }
  mc::after_previous();
  if (!on) return;
  const float2 a = run.sum(d, d.s_tmp);
  d.uc[c] = make_float2(u.x + a.x * iv, u.y + a.y * iv);
}
__global__ void k_ib_rev_node(AD d, int it) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  switch (d.KK) {
    case 16: return rev_node<16>(d, n, it);
    case 9: return rev_node<9>(d, n, it);
    case 4: return rev_node<4>(d, n, it);
    default: return rev_node<0>(d, n, it);
  }
}
__global__ void k_ib_rev_cell(AD d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < __ldcg(d.ntouched);
  CellRun run;
  int c = 0;
  if (on) {
    c = __ldcg(d.touched + i);
    run.load(d, c);
  }
  mc::after_previous();
  if (!on) return;
  const float2 a = run.sum(d, d.s_tmp);
  const float2 u = d.luc[c];
  d.luc[c] = make_float2(u.x + a.x, u.y + a.y);
}

// ------------------------------------------------------------------ adjoint: stream + collide + F
__constant__ float kW9[9] = {4.0f / 9.0f, 1.0f / 9.0f, 1.0f / 9.0f, 1.0f / 9.0f, 1.0f / 9.0f,
                             1.0f / 36.0f, 1.0f / 36.0f, 1.0f / 36.0f, 1.0f / 36.0f};
// opposite D2Q9 direction {0, 3, 4, 1, 2, 7, 8, 5, 6} as a compile-time function: in the
// unrolled population loops the index folds to a constant and the per-cell arrays stay in
// registers (a table lookup would put them in local memory)
__device__ __forceinline__ constexpr int opp9(int i) { return i == 0 ? 0 : (i <= 4 ? (i + 1) % 4 + 1 : (i - 3) % 4 + 5); }

__global__ void k_lbm_adj1(AD d) {
  mc::after_previous();
  const StepArgs a = d.sa[*d.jp];
  const float* __restrict__ f = a.f;
  const float* __restrict__ lfn = a.lf_in;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.lHW) return;
  const int y = c / d.lW, x = c - y * d.lW;
  float f0[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) f0[i] = mc::max_prop(f[(size_t)i * d.lHW + c], MC_EPSIL);
  float rr = f0[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) rr = rr + f0[i];
  const float rho = mc::max_prop(rr, 0.1f);
  const float ux = ((((f0[1] - f0[3]) + f0[5]) - f0[6]) - f0[7]) + f0[8];
  const float uy = ((((f0[2] - f0[4]) + f0[5]) + f0[6]) - f0[7]) - f0[8];
  const float c1 = mc::clamp_factor(ux / rho, uy / rho, d.vmax);
  const float vx = (ux / rho) * c1, vy = (uy / rho) * c1;
  const float2 u5 = d.uc[c];
  const float u5x = u5.x, u5y = u5.y;
  const float c2 = mc::clamp_factor(u5x, u5y, d.vmax);
  const float ucx = u5x * c2, ucy = u5y * c2;
  const float Frx = (ucx - vx) * rho, Fry = (ucy - vy) * rho;
  float Fx = Frx, Fy = Fry;
  if (d.force_clamp) {
    const float c3 = mc::clamp_factor(Frx, Fry, d.vmax);
    Fx = Frx * c3;
    Fy = Fry * c3;
  }
  // forward collide for the floor masks
  float post[9], us_x, us_y;
  mc::collide(f0, rho, vx, vy, Fx, Fy, d.wp, d.wm, d.cp, d.cm, post, us_x, us_y);
  // recompute the unfloored collide output for the first mask
  const float half = 0.5f;
  const float usx = vx + half * Fx / rho, usy = vy + half * Fy / rho;
  const float usq = usx * usx + usy * usy;
  const float udF = usx * Fx + usy * Fy;
  float eu[9], eF[9], feq[9], raw[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    eu[i] = (float)mc::kEx[i] * usx + (float)mc::kEy[i] * usy;
    eF[i] = (float)mc::kEx[i] * Fx + (float)mc::kEy[i] * Fy;
    feq[i] = (rho * kW9[i]) * (((1.0f + 3.0f * eu[i]) + 4.5f * (eu[i] * eu[i])) - 1.5f * usq);
    raw[i] = kW9[i] * (3.0f * (eF[i] - udF) + (9.0f * eu[i]) * eF[i]);
  }
  float g[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int o = opp9(i);
    const float pr = f0[i] - d.wp * (half * (f0[i] + f0[o]) - half * (feq[i] + feq[o])) -
                     d.wm * (half * (f0[i] - f0[o]) - half * (feq[i] - feq[o]));
    const float src = d.cp * (half * (raw[i] + raw[o])) + d.cm * (half * (raw[i] - raw[o]));
    const int xn = x + mc::kEx[i], yn = y + mc::kEy[i];
    const float lin = lfn[(size_t)i * d.lHW + cell_of(yn, xn, d.lH, d.lW)];
    g[i] = (lin * dmaxf(post[i], MC_EPSIL)) * dmaxf(pr + src, MC_EPSIL);
  }
  float lf0[9];
  float lrho = 0.0f, lusx = 0.0f, lusy = 0.0f, lFx = 0.0f, lFy = 0.0f;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int o = opp9(i);
    const float gp = half * (g[i] + g[o]), gm = half * (g[i] - g[o]);
    lf0[i] = g[i] - d.wp * gp - d.wm * gm;
    const float lfeq = d.wp * gp + d.wm * gm;
    const float lraw = (1.0f - half * d.wp) * gp + (1.0f - half * d.wm) * gm;
    const float ex = (float)mc::kEx[i], ey = (float)mc::kEy[i];
    lrho += lfeq * kW9[i] * (1.0f + 3.0f * eu[i] + 4.5f * eu[i] * eu[i] - 1.5f * usq);
    const float a = lfeq * rho * kW9[i];
    lusx += a * (3.0f * ex + 9.0f * eu[i] * ex - 3.0f * usx);
    lusy += a * (3.0f * ey + 9.0f * eu[i] * ey - 3.0f * usy);
    const float b = lraw * kW9[i];
    lusx += b * (-3.0f * Fx + 9.0f * eF[i] * ex);
    lusy += b * (-3.0f * Fy + 9.0f * eF[i] * ey);
    lFx += b * (3.0f * ex - 3.0f * usx + 9.0f * eu[i] * ex);
    lFy += b * (3.0f * ey - 3.0f * usy + 9.0f * eu[i] * ey);
  }
  float lvx = lusx, lvy = lusy;
  lFx += half * lusx / rho;
  lFy += half * lusy / rho;
  lrho -= half * (lusx * Fx + lusy * Fy) / (rho * rho);
  // node reaction: vel_out = vel1 - (nf / m) / sdt, nf = sum_s w F[idx] (with synthetic
  // pairs, nf of a node = 0.5 (nf of its + point + nf of its - point))
  const bool syn = d.NI > d.N;
  float rx = 0.0f, ry = 0.0f;
  const int len = d.cnt[c], first = len > 0 ? d.start[c] : 0;
  for (int q = first; q < first + len; ++q) {
    const int e = d.ent[q];
    const float w = d.ib_w[e];
    const int pt = e / d.KK;
    const float2 lv = d.lvel[pt < d.N ? pt : pt - d.N];
    float gx = (-lv.x / d.mass) / d.sdtx, gy = (-lv.y / d.mass) / d.sdty;
    if (syn) {
      gx = 0.5f * gx;
      gy = 0.5f * gy;
    }
    rx = rx + w * gx;
    ry = ry + w * gy;
  }
  lFx = rx + lFx;
  lFy = ry + lFy;
  if (d.force_clamp) {
    const float2 lr = clamp_vjp(Frx, Fry, d.vmax, lFx, lFy);
    lFx = lr.x;
    lFy = lr.y;
  }
  // F = (ucc - v) rho
  const float lccx = lFx * rho, lccy = lFy * rho;
  lvx -= lFx * rho;
  lvy -= lFy * rho;
  lrho += lFx * (ucx - vx) + lFy * (ucy - vy);  // through F_raw = (ucc - v) rho
  const float2 l5 = clamp_vjp(u5x, u5y, d.vmax, lccx, lccy);
  d.luc[c] = l5;
  d.lv[c] = lvx;
  d.lv[d.lHW + c] = lvy;
  d.lrho[c] = lrho;
#pragma unroll
  for (int i = 0; i < 9; ++i) d.lf0p[(size_t)i * d.lHW + c] = lf0[i];
}

__global__ void k_lbm_adj2(AD d) {
  mc::after_previous();
  const StepArgs a = d.sa[*d.jp];
  const float* __restrict__ f = a.f;
  float* __restrict__ lf_out = a.lf_out;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.lHW) return;
  float f0[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) f0[i] = mc::max_prop(f[(size_t)i * d.lHW + c], MC_EPSIL);
  float rr = f0[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) rr = rr + f0[i];
  const float rho = mc::max_prop(rr, 0.1f);
  const float ux = (((((f0[1] - f0[3]) + f0[5]) - f0[6]) - f0[7]) + f0[8]) / rho;
  const float uy = (((((f0[2] - f0[4]) + f0[5]) + f0[6]) - f0[7]) - f0[8]) / rho;
  const float2 lu5 = d.luc[c];
  const float lvx = d.lv[c] + lu5.x, lvy = d.lv[d.lHW + c] + lu5.y;
  d.cnt[c] = 0;  // the lattice's entries have been used
  const float2 lu = clamp_vjp(ux, uy, d.vmax, lvx, lvy);
  const float lrho = d.lrho[c] - (lu.x * ux + lu.y * uy) / rho;
  const float lraw = lrho * dmaxf(rr, 0.1f);
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const float l0 = d.lf0p[(size_t)i * d.lHW + c] + lraw + ((float)mc::kEx[i] * lu.x + (float)mc::kEy[i] * lu.y) / rho;
    lf_out[(size_t)i * d.lHW + c] = l0 * dmaxf(f[(size_t)i * d.lHW + c], MC_EPSIL);
  }
}

// ------------------------------------------------------------------ adjoint: node velocity / position
__global__ void k_node_adj(AD d) {
  mc::after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 3) d.ntouched[i] = 0;
  if (i < d.E) d.lt[0][i] = d.lth[i];
  if (i >= d.N) return;
  float2 lv1 = d.lvel[i];
  if (d.fluid) {
    float2 a = d.lnv[i];
    if (d.NI > d.N) {  // both synthetic points carry the node's velocity
      const float2 b = d.lnv[i + d.N];
      a.x = a.x + b.x;
      a.y = a.y + b.y;
    }
    lv1.x = lv1.x + (a.x * d.scx) * d.dt;
    lv1.y = lv1.y + (a.y * d.scy) * d.dt;
  }
  const float2 lp = d.lpos[i];
  d.lp[0][i] = make_float2(lp.x + lv1.x / d.dt, lp.y + lv1.y / d.dt);
  d.lprev[i] = make_float2(-lv1.x / d.dt, -lv1.y / d.dt);
}

// ------------------------------------------------------------------ adjoint: PBD iterations (one CTA per rod component)
// The reverse iterations of a component whose edges, nodes and bending pairs fit one per
// thread (kPbdGather incidences at most): topology in registers, the accumulated cotangents
// of the owned edge / pair (d_len, rest_acc, d_kb) in registers and written once.  Same
// arithmetic and order as the general loops of k_pbd_rev.  All threads of the CTA call it;
// false (nothing done) when the component does not fit.
__device__ __forceinline__ bool pbd_rev_fast(const AD& d, int ea, int eb, int na, int nb, int ba, int bb, float ks,
                                             float kst) {
  const int tid = threadIdx.x;
  PbdNodeReg rn;
  int e = -1, ne3 = 0, b = -1;
  int2 pr = make_int2(0, 0), bp = make_int2(0, 0);
  float ns = 1.0f, nt = 1.0f, L0 = 0.0f, ed_x = 1.0f, ed_y = 1.0f, kbb = 0.0f, rst = 0.0f;
  int bq[kPbdGather];
  bool negq[kPbdGather];
  bool ok = eb - ea <= kPbdRod && nb - na <= kPbdRod && bb - ba <= kPbdRod;
  if (ok) ok = pbd_load_node(d, na + tid, nb, rn);
  if (ok && ea + tid < eb) {
    e = d.c_edges[ea + tid];
    pr = d.pairs[e];
    ns = d.ndeg[pr.x];
    nt = d.ndeg[pr.y];
    L0 = d.rest_len[e];
    const int qa = d.e_start[e];
    ne3 = d.e_start[e + 1] - qa;
    if (ne3 > kPbdGather) ok = false;
#pragma unroll
    for (int q = 0; q < kPbdGather; ++q)
      if (q < ne3) {
        const int en = d.e_list[qa + q];
        bq[q] = en >> 1;
        negq[q] = en & 1;
      }
  }
  if (ok && ba + tid < bb) {
    b = d.c_bps[ba + tid];
    bp = d.bpairs[b];
    ed_x = d.edeg[bp.x];
    ed_y = d.edeg[bp.y];
    kbb = d.kb[b];
    rst = d.rest[b];
  }
  // places in the component instead of global indices
  int2 prl = make_int2(0, 0), bpl = make_int2(0, 0);
  if (ok && rn.n >= 0) {
#pragma unroll
    for (int q = 0; q < kPbdGather; ++q)
      if (q < rn.ne) rn.e[q] = local_of(d.c_edges, ea, eb, rn.e[q]);
  }
  if (ok && e >= 0) {
    prl = make_int2(local_of(d.c_nodes, na, nb, pr.x), local_of(d.c_nodes, na, nb, pr.y));
#pragma unroll
    for (int q = 0; q < kPbdGather; ++q)
      if (q < ne3) {
        bq[q] = local_of(d.c_bps, ba, bb, bq[q]);
        if (bq[q] < 0) ok = false;
      }
  }
  if (ok && b >= 0) {
    bpl = make_int2(local_of(d.c_edges, ea, eb, bp.x), local_of(d.c_edges, ea, eb, bp.y));
    if (bpl.x < 0 || bpl.y < 0) ok = false;
  }
  if (!__syncthreads_and(ok)) return false;
  __shared__ float2 lp[kPbdRod], lcur[kPbdRod];
  __shared__ float lthn[kPbdRod], gb[kPbdRod], l0s[kPbdRod];
  __shared__ int2 ends[kPbdRod];
  // per (iteration, edge): segment, (L - L0) / m and its derivative, m, the new angle's cosine and
  // sine; per (iteration, pair): deviation from the rest angle
  __shared__ float2 seg[kRevChunk][kPbdRod], stretch[kRevChunk][kPbdRod], turn[kRevChunk][kPbdRod];
  __shared__ float length[kRevChunk][kPbdRod], bend[kRevChunk][kPbdRod];
  const int ne = eb - ea;
  if (rn.n >= 0) lp[tid] = d.lp[0][rn.n];
  if (e >= 0) {
    ends[tid] = pr;
    l0s[tid] = L0;
  }
  float acc_len = e >= 0 ? d.d_len[e] : 0.0f, lt = e >= 0 ? d.lt[0][e] : 0.0f;
  float acc_rest = b >= 0 ? d.rest_acc[b] : 0.0f;
  float acc_kb = b >= 0 ? d.d_kb[b] : 0.0f;
  const float rns = 1.0f / ns, rnt = 1.0f / nt, red_x = 1.0f / ed_x, red_y = 1.0f / ed_y;
  __syncthreads();
  for (int k1 = d.C; k1 > 0; k1 -= kRevChunk) {
    const int k0 = max(k1 - kRevChunk, 0);
    for (int k = k0 + (tid >> 5); k < k1; k += kPbdThreads / 32) {
      const float2* p = d.pp + (size_t)k * d.N;
      const float* thn = d.tt + (size_t)(k + 1) * d.E;
      for (int i = tid & 31; i < ne; i += 32) {
        const int2 g = ends[i];
        const float2 pa = p[g.x], pb = p[g.y];
        const float th_n = thn[d.c_edges[ea + i]], l0 = l0s[i];
        const float2 cur_v = mc::min_image(pb.x, pb.y, pa.x, pa.y, (float)d.W, (float)d.H);
        const float L = sqrtf(cur_v.x * cur_v.x + cur_v.y * cur_v.y);
        const float m = mc::max_prop(L, 1e-8f);
        float cs, sn;
        sincosf(th_n, &sn, &cs);
        seg[k - k0][i] = cur_v;
        stretch[k - k0][i] = make_float2((L - l0) / m, (1.0f / m - (L - l0) * dmaxf(L, 1e-8f) / (m * m)) / L);
        length[k - k0][i] = m;
        turn[k - k0][i] = make_float2(cs, sn);
      }
    }
    if (b >= 0) {
      const float pi = (float)M_PI;
      for (int k = k0; k < k1; ++k) {
        const float* th = d.tt + (size_t)k * d.E;
        const float diff = mc::fmod_floor((th[bp.y] - th[bp.x]) + pi, (float)(2.0 * M_PI)) - pi;
        bend[k - k0][tid] = diff - rst;
      }
    }
    __syncthreads();
    for (int k = k1 - 1 - k0; k >= 0; --k) {
      // position pass
      float lthn_e = 0.0f;
      if (e >= 0) {
        const float2 la = lp[prl.x], lb = lp[prl.y], cur_v = seg[k][tid], st = stretch[k][tid], cssn = turn[k][tid];
        const float hx = ((div_degree(la.x, ns, rns) - div_degree(lb.x, nt, rnt)) * kst) * 0.5f;
        const float hy = ((div_degree(la.y, ns, rns) - div_degree(lb.y, nt, rnt)) * kst) * 0.5f;
        const float a = st.x, da = st.y;
        const float lsx = (1.0f - ks) * hx, lsy = (1.0f - ks) * hy;
        const float sdot = cur_v.x * lsx + cur_v.y * lsy;
        const float lcx = ks * hx + a * lsx + (sdot * da) * cur_v.x;
        const float lcy = ks * hy + a * lsy + (sdot * da) * cur_v.y;
        const float ltx = -ks * hx, lty = -ks * hy;
        const float cs = cssn.x, sn = cssn.y;
        acc_len += -sdot / length[k][tid] + (cs * ltx + sn * lty);
        lthn_e = lt + L0 * (-sn * ltx + cs * lty);
        lthn[tid] = lthn_e;
        lcur[tid] = make_float2(lcx, lcy);
      }
      __syncthreads();
      if (rn.n >= 0) {
        float2 a = lp[tid];
#pragma unroll
        for (int q = 0; q < kPbdGather; ++q)
          if (q < rn.ne) {
            const float2 lc = lcur[rn.e[q]];
            if (rn.neg[q]) {
              a.x += lc.x;
              a.y += lc.y;
            } else {
              a.x -= lc.x;
              a.y -= lc.y;
            }
          }
        lp[tid] = a;
      }
      if (b >= 0) {
        const float lcorr =
            1.8f * (div_degree(lthn[bpl.x], ed_x, red_x) - div_degree(lthn[bpl.y], ed_y, red_y));
        const float g = lcorr * kbb * 0.5f;
        gb[tid] = g;
        acc_rest -= g;
        acc_kb += lcorr * bend[k][tid] * 0.5f;
      }
      __syncthreads();
      if (e >= 0) {
        float a = lthn_e;
#pragma unroll
        for (int q = 0; q < kPbdGather; ++q)
          if (q < ne3) a += negq[q] ? gb[bq[q]] : -gb[bq[q]];
        lt = a;
      }
    }
    __syncthreads();
  }
  if (rn.n >= 0) d.lp[d.C & 1][rn.n] = lp[tid];
  if (e >= 0) d.lt[d.C & 1][e] = lt;
  if (e >= 0) d.d_len[e] = acc_len;
  if (b >= 0) {
    d.rest_acc[b] = acc_rest;
    d.d_kb[b] = acc_kb;
  }
  __syncthreads();
  return true;
}

__global__ void __launch_bounds__(kPbdThreads) k_pbd_rev(AD d) {
  mc::after_previous();
  const int t = d.sa[*d.jp].t;
  const int c = blockIdx.x;
  const int ea = d.c_estart[c], eb = d.c_estart[c + 1], na = d.c_nstart[c], nb = d.c_nstart[c + 1];
  const int ba = d.c_bstart[c], bb = d.c_bstart[c + 1];
  int cur = 0;
  const float ks = d.kshear, kst = d.kstretch;
  if (pbd_rev_fast(d, ea, eb, na, nb, ba, bb, ks, kst))
    cur = d.C & 1;
  else
  for (int k = d.C - 1; k >= 0; --k) {
    const float2* p = d.pp + (size_t)k * d.N;
    const float* th = d.tt + (size_t)k * d.E;
    const float* thn = d.tt + (size_t)(k + 1) * d.E;
    const float2* lpi = d.lp[cur];
    float2* lpo = d.lp[cur ^ 1];
    const float* lti = d.lt[cur];
    float* lto = d.lt[cur ^ 1];
    // position pass
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      const int2 pr = d.pairs[e];
      const float ns = d.ndeg[pr.x], nt = d.ndeg[pr.y];
      const float hx = ((lpi[pr.x].x / ns - lpi[pr.y].x / nt) * kst) * 0.5f;
      const float hy = ((lpi[pr.x].y / ns - lpi[pr.y].y / nt) * kst) * 0.5f;
      const float2 cur_v = mc::min_image(p[pr.y].x, p[pr.y].y, p[pr.x].x, p[pr.x].y, (float)d.W, (float)d.H);
      const float L = sqrtf(cur_v.x * cur_v.x + cur_v.y * cur_v.y);
      const float L0 = d.rest_len[e];
      const float m = mc::max_prop(L, 1e-8f);
      const float a = (L - L0) / m;
      const float da = (1.0f / m - (L - L0) * dmaxf(L, 1e-8f) / (m * m)) / L;
      const float lsx = (1.0f - ks) * hx, lsy = (1.0f - ks) * hy;
      const float sdot = cur_v.x * lsx + cur_v.y * lsy;
      const float lcx = ks * hx + a * lsx + (sdot * da) * cur_v.x;
      const float lcy = ks * hy + a * lsy + (sdot * da) * cur_v.y;
      const float ltx = -ks * hx, lty = -ks * hy;
      float cs, sn;
      sincosf(thn[e], &sn, &cs);
      d.d_len[e] += -sdot / m + (cs * ltx + sn * lty);
      d.lthn[e] = lti[e] + L0 * (-sn * ltx + cs * lty);
      d.lcur[e] = make_float2(lcx, lcy);
    }
    __syncthreads();
    for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
      const int n = d.c_nodes[in];
      float ax = lpi[n].x, ay = lpi[n].y;
      for (int q = d.n_start[n]; q < d.n_start[n + 1]; ++q) {
        const int en = d.n_list[q];
        const float2 lc = d.lcur[en >> 1];
        if (en & 1) {
          ax += lc.x;
          ay += lc.y;
        } else {
          ax -= lc.x;
          ay -= lc.y;
        }
      }
      lpo[n] = make_float2(ax, ay);
    }
    for (int ib = ba + threadIdx.x; ib < bb; ib += blockDim.x) {
      const int b = d.c_bps[ib];
      const int2 bp = d.bpairs[b];
      const float lcorr = 1.8f * (d.lthn[bp.x] / d.edeg[bp.x] - d.lthn[bp.y] / d.edeg[bp.y]);
      const float g = lcorr * d.kb[b] * 0.5f;
      d.gb[b] = g;
      d.rest_acc[b] -= g;
      const float pi = (float)M_PI;
      const float diff = mc::fmod_floor((th[bp.y] - th[bp.x]) + pi, (float)(2.0 * M_PI)) - pi;
      d.d_kb[b] += lcorr * (diff - d.rest[b]) * 0.5f;
    }
    __syncthreads();
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      float a = d.lthn[e];
      for (int q = d.e_start[e]; q < d.e_start[e + 1]; ++q) {
        const int en = d.e_list[q];
        const float g = d.gb[en >> 1];
        a += (en & 1) ? g : -g;
      }
      lto[e] = a;
    }
    __syncthreads();
    cur ^= 1;
  }
  for (int in = na + threadIdx.x; in < nb; in += blockDim.x) d.lpred1[d.c_nodes[in]] = d.lp[cur][d.c_nodes[in]];
  for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) d.lth[d.c_edges[ie]] = d.lt[cur][d.c_edges[ie]];
  for (int ib = ba + threadIdx.x; ib < bb; ib += blockDim.x) {
    const int b = d.c_bps[ib];
    const float G = d.rest_acc[b];
    if (d.has_act) {
      const float arg = d.act_om[b] * (float)t + d.act_ph[b];
      float sn, cs;
      sincosf(arg, &sn, &cs);
      d.d_c[b] += G;
      d.d_amp[b] += G * sn;
      d.d_ph[b] += G * d.act_amp[b] * cs;
      d.d_om[b] += G * d.act_amp[b] * cs * (float)t;
    } else {
      d.d_rest[b] += G;
    }
  }
}

// ------------------------------------------------------------------ stable-Cosserat iterations
// (solver/stable_cosserat.py:13-119), one CTA per rod component like the PBD kernels.
// Iteration k: theta' = pull(theta + sum(+-corr) / edeg) toward the segment direction,
// then x' = x + (w (y - x) + sum(+-f_e)) / (w + sum k_s / l_e^2) with
// f_e = (k_s / l_e)(r_e / l_e - (cos theta'_e, sin theta'_e)), r_e the min-image segment,
// y the prediction (pp[0]).  Same arithmetic and sum order as the forward rod kernels.
__device__ __forceinline__ float2 cos_force(const AD& d, const float2* p, float thn, int e) {
  const int2 pr = d.pairs[e];
  const float L0 = d.rest_len[e];
  const float2 r = mc::min_image(p[pr.y].x, p[pr.y].y, p[pr.x].x, p[pr.x].y, (float)d.W, (float)d.H);
  float sn, cs;
  sincosf(thn, &sn, &cs);
  const float kl = d.kstretch / L0;
  return make_float2(kl * (r.x / L0 - cs), kl * (r.y / L0 - sn));
}

// the summed force and stiffness of node n at iterate p, angles thn
__device__ __forceinline__ void cos_node_sum(const AD& d, const float2* p, const float* thn, int n, float& ax,
                                             float& ay, float& hh) {
  const float w = d.cos_w;
  ax = w * (d.pp[n].x - p[n].x);
  ay = w * (d.pp[n].y - p[n].y);
  hh = w;
  for (int q = d.n_start[n]; q < d.n_start[n + 1]; ++q) {
    const int en = d.n_list[q];
    const int e = en >> 1;
    const float2 f = cos_force(d, p, thn[e], e);
    if (en & 1) {
      ax = ax + (-f.x);
      ay = ay + (-f.y);
    } else {
      ax = ax + f.x;
      ay = ay + f.y;
    }
    const float L0 = d.rest_len[e];
    hh = hh + d.kstretch / (L0 * L0);
  }
}

__global__ void __launch_bounds__(kPbdThreads) k_cos_fwd(AD d) {
  mc::after_previous();
  const int c = blockIdx.x;
  const int ea = d.c_estart[c], eb = d.c_estart[c + 1], na = d.c_nstart[c], nb = d.c_nstart[c + 1];
  for (int k = 0; k < d.C; ++k) {
    const float* th = d.tt + (size_t)k * d.E;
    float* thn = d.tt + (size_t)(k + 1) * d.E;
    const float2* p = d.pp + (size_t)k * d.N;
    float2* pn = d.pp + (size_t)(k + 1) * d.N;
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      float acc = 0.0f;
      for (int q = d.e_start[e]; q < d.e_start[e + 1]; ++q) {
        const int en = d.e_list[q];
        const float cr = bend_corr(d, th, en >> 1);
        acc = acc + ((en & 1) ? -cr : cr);
      }
      const int2 pr = d.pairs[e];
      const float2 r = mc::min_image(p[pr.y].x, p[pr.y].y, p[pr.x].x, p[pr.x].y, (float)d.W, (float)d.H);
      thn[e] = mc::cos_pull(th[e] + acc / d.edeg[e], r.x, r.y);
    }
    __syncthreads();
    for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
      const int n = d.c_nodes[in];
      float ax, ay, hh;
      cos_node_sum(d, p, thn, n, ax, ay, hh);
      pn[n] = make_float2(p[n].x + ax / hh, p[n].y + ay / hh);
    }
    __syncthreads();
  }
}

// Reverse of k_cos_fwd.  mod passes its cotangent through (derivative 1) and
// d atan2(r_y, r_x) = (r_x dr_y - r_y dr_x) / |r|^2.
__global__ void __launch_bounds__(kPbdThreads) k_cos_rev(AD d) {
  mc::after_previous();
  const int t = d.sa[*d.jp].t;
  const int c = blockIdx.x;
  const int ea = d.c_estart[c], eb = d.c_estart[c + 1], na = d.c_nstart[c], nb = d.c_nstart[c + 1];
  const int ba = d.c_bstart[c], bb = d.c_bstart[c + 1];
  const float ks = d.kstretch, w = d.cos_w;
  int cur = 0;
  for (int in = na + threadIdx.x; in < nb; in += blockDim.x) d.ly[d.c_nodes[in]] = make_float2(0.0f, 0.0f);
  for (int k = d.C - 1; k >= 0; --k) {
    const float2* p = d.pp + (size_t)k * d.N;
    const float* th = d.tt + (size_t)k * d.E;
    const float* thn = d.tt + (size_t)(k + 1) * d.E;
    const float2* lpi = d.lp[cur];
    float2* lpo = d.lp[cur ^ 1];
    const float* lti = d.lt[cur];
    float* lto = d.lt[cur ^ 1];
    // x' = x + F / h: cotangents of F, h, y and the direct part of x
    for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
      const int n = d.c_nodes[in];
      float ax, ay, hh;
      cos_node_sum(d, p, thn, n, ax, ay, hh);
      const float2 lx = lpi[n];
      const float lfx = lx.x / hh, lfy = lx.y / hh;
      d.lfn[n] = make_float2(lfx, lfy);
      d.lhn[n] = -(lx.x * ax + lx.y * ay) / (hh * hh);
      const float2 yy = d.ly[n];
      d.ly[n] = make_float2(yy.x + w * lfx, yy.y + w * lfy);
      lpo[n] = make_float2(lx.x - w * lfx, lx.y - w * lfy);
    }
    __syncthreads();
    // per edge: f_e and h_e -> segment, angle, rest length; then the pull
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      const int2 pr = d.pairs[e];
      const float L0 = d.rest_len[e];
      const float2 r = mc::min_image(p[pr.y].x, p[pr.y].y, p[pr.x].x, p[pr.x].y, (float)d.W, (float)d.H);
      float sn, cs;
      sincosf(thn[e], &sn, &cs);
      const float2 a = d.lfn[pr.x], b = d.lfn[pr.y];
      const float lfx = a.x - b.x, lfy = a.y - b.y;
      const float kl = ks / L0;
      float lrx = (kl / L0) * lfx, lry = (kl / L0) * lfy;
      const float lthn = lti[e] + kl * (lfx * sn - lfy * cs);
      const float cx = r.x / L0 - cs, cy = r.y / L0 - sn;
      d.d_len[e] += -(kl / L0) * (lfx * cx + lfy * cy) - (kl / (L0 * L0)) * (lfx * r.x + lfy * r.y) +
                    (d.lhn[pr.x] + d.lhn[pr.y]) * (-2.0f * ks / (L0 * L0 * L0));
      const float la = 0.05f * lthn;
      const float r2 = r.x * r.x + r.y * r.y;
      lrx += -r.y * la / r2;
      lry += r.x * la / r2;
      d.lcur[e] = make_float2(lrx, lry);
      d.lthn[e] = lthn - 0.05f * lthn;  // cotangent of the angle before the pull
    }
    __syncthreads();
    for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
      const int n = d.c_nodes[in];
      float ax = lpo[n].x, ay = lpo[n].y;
      for (int q = d.n_start[n]; q < d.n_start[n + 1]; ++q) {
        const int en = d.n_list[q];
        const float2 lc = d.lcur[en >> 1];
        if (en & 1) {
          ax += lc.x;
          ay += lc.y;
        } else {
          ax -= lc.x;
          ay -= lc.y;
        }
      }
      lpo[n] = make_float2(ax, ay);
    }
    for (int ib = ba + threadIdx.x; ib < bb; ib += blockDim.x) {
      const int b = d.c_bps[ib];
      const int2 bp = d.bpairs[b];
      const float lcorr = d.lthn[bp.x] / d.edeg[bp.x] - d.lthn[bp.y] / d.edeg[bp.y];
      const float g = lcorr * d.kb[b] * 0.5f;
      d.gb[b] = g;
      d.rest_acc[b] -= g;
      const float pi = (float)M_PI;
      const float diff = mc::fmod_floor((th[bp.y] - th[bp.x]) + pi, (float)(2.0 * M_PI)) - pi;
      d.d_kb[b] += lcorr * (diff - d.rest[b]) * 0.5f;
    }
    __syncthreads();
    for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) {
      const int e = d.c_edges[ie];
      float a = d.lthn[e];
      for (int q = d.e_start[e]; q < d.e_start[e + 1]; ++q) {
        const int en = d.e_list[q];
        const float g = d.gb[en >> 1];
        a += (en & 1) ? g : -g;
      }
      lto[e] = a;
    }
    __syncthreads();
    cur ^= 1;
  }
  // the iterations start from the prediction and are pulled toward it
  for (int in = na + threadIdx.x; in < nb; in += blockDim.x) {
    const int n = d.c_nodes[in];
    const float2 a = d.lp[cur][n], yy = d.ly[n];
    d.lpred1[n] = make_float2(a.x + yy.x, a.y + yy.y);
  }
  for (int ie = ea + threadIdx.x; ie < eb; ie += blockDim.x) d.lth[d.c_edges[ie]] = d.lt[cur][d.c_edges[ie]];
  for (int ib = ba + threadIdx.x; ib < bb; ib += blockDim.x) {
    const int b = d.c_bps[ib];
    const float G = d.rest_acc[b];
    if (d.has_act) {
      const float arg = d.act_om[b] * (float)t + d.act_ph[b];
      float sn, cs;
      sincosf(arg, &sn, &cs);
      d.d_c[b] += G;
      d.d_amp[b] += G * sn;
      d.d_ph[b] += G * d.act_amp[b] * cs;
      d.d_om[b] += G * d.act_amp[b] * cs * (float)t;
    } else {
      d.d_rest[b] += G;
    }
  }
}

// ------------------------------------------------------------------ adjoint: steric
__device__ __forceinline__ void sample_adj(const AD& d, const float* V, float yy, float xx, float coef, int n, int qs,
                                           float& lpx, float& lpy) {
  const float ly = floorf(yy), lx = floorf(xx);
  const float ty = yy - ly, tx = xx - lx;
  const int iy = (int)ly, ix = (int)lx;
  const int y0 = mc::imod_floor(iy, d.H), y1 = mc::imod_floor(iy + 1, d.H);
  const int x0 = mc::imod_floor(ix, d.W), x1 = mc::imod_floor(ix + 1, d.W);
  const float v00 = V[y0 * d.W + x0], v01 = V[y0 * d.W + x1], v10 = V[y1 * d.W + x0], v11 = V[y1 * d.W + x1];
  lpx = coef * ((1.0f - ty) * (v01 - v00) + ty * (v11 - v10));
  lpy = coef * ((1.0f - tx) * (v10 - v00) + tx * (v11 - v01));
  const int base = n * 16 + qs * 4;
  d.st_val[base + 0] = coef * ((1.0f - ty) * (1.0f - tx));
  d.st_val[base + 1] = coef * ((1.0f - ty) * tx);
  d.st_val[base + 2] = coef * (ty * (1.0f - tx));
  d.st_val[base + 3] = coef * (ty * tx);
  cell_append(d, y0 * d.W + x0, base);
  cell_append(d, y0 * d.W + x1, base + 1);
  cell_append(d, y1 * d.W + x0, base + 2);
  cell_append(d, y1 * d.W + x1, base + 3);
}

// 4 lanes per node: lane q one of the four bilinear samples and a quarter of the neighbours; the
// terms are added in the order samples, then neighbours.  384 nodes: 12.6 -> 7.6 us against one
// thread per node.
__global__ void __launch_bounds__(128) k_steric_adj_node(AD d) {
  mc::after_previous();
  const float* __restrict__ V = d.sa[*d.jp].V;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = min(t >> 2, d.N - 1), qs = t & 3;
  const bool on = (t >> 2) < d.N;
  const unsigned full = 0xffffffffu;
  const float Wf = (float)d.W, Hf = (float)d.H;
  const float2 lp1 = d.lpred1[n];
  const float lfx = (lp1.x * d.st_strength) * d.dt, lfy = (lp1.y * d.st_strength) * d.dt;
  const float2 q = d.pred0[n];
  const float x = mc::fmod_floor(q.x, Wf), y = mc::fmod_floor(q.y, Hf);
  const float e = 0.5f;
  float tx = 0.0f, ty = 0.0f;
  if (on)
    sample_adj(d, V, qs < 2 ? y : (qs == 2 ? y + e : y - e), qs > 1 ? x : (qs == 0 ? x + e : x - e),
               qs == 0 ? -lfx : qs == 1 ? lfx : qs == 2 ? -lfy : lfy, n, qs, tx, ty);
  float lpx = 0.0f, lpy = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    lpx += __shfl_sync(full, tx, i, 4);
    lpy += __shfl_sync(full, ty, i, 4);
  }
  if (d.nskip > 0) {
    const float s2 = d.sigma * d.sigma;
    const float inv2s2 = 2.0f * d.sigma * d.sigma;
    const float norm = (float)(2.0 * M_PI) * d.sigma * d.sigma;
    const float pre = d.scatter / (d.sigma * d.sigma);
    for (int o0 = -d.nskip; o0 <= d.nskip; o0 += 4) {
      const int o = o0 + qs, j = n + o;
      const bool there = o != 0 && o <= d.nskip && j >= 0 && j < d.N;
      tx = ty = 0.0f;
      if (there) {
        const float2 qj = d.pred0[j];
        const float2 r = mc::min_image(x, y, mc::fmod_floor(qj.x, Wf), mc::fmod_floor(qj.y, Hf), Wf, Hf);
        const float d2 = r.x * r.x + r.y * r.y;
        const float K = expf(-d2 / inv2s2) / norm;
        const float2 lpj = d.lpred1[j];
        const float ljx = (lpj.x * d.st_strength) * d.dt, ljy = (lpj.y * d.st_strength) * d.dt;
        // J(r) (g_n - g_j) with g = -pre * lf and J = K (I - r r^T / sigma^2)
        const float gx = -pre * (lfx - ljx), gy = -pre * (lfy - ljy);
        const float rg = (r.x * gx + r.y * gy) / s2;
        tx = K * (gx - r.x * rg);
        ty = K * (gy - r.y * rg);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        lpx += __shfl_sync(full, tx, i, 4);
        lpy += __shfl_sync(full, ty, i, 4);
      }
    }
  }
  if (on && qs == 0) d.lpred0p[n] = make_float2(lp1.x + lpx, lp1.y + lpy);
}

// out must be zero outside the touched cells
__global__ void k_gather_field(AD d, const float* val, float* out) {
  mc::after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *d.ntouched) return;
  const int c = d.touched[i];
  float a = 0.0f;
  for (int q = d.start[c], end = q + d.cnt[c]; q < end; ++q) a = a + val[d.ent[q]];
  out[c] = a;
  d.cnt[c] = 0;  // used
}

__global__ void k_steric_adj_cic(AD d) {
  mc::after_previous();
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= d.N) return;
  float2 l0 = d.lpred0p[n];
  if (d.steric) {
    const float Wf = (float)d.W, Hf = (float)d.H;
    const float2 q = d.pred0[n];
    const float x = mc::fmod_floor(q.x, Wf), y = mc::fmod_floor(q.y, Hf);
    const float fx = floorf(x), fy = floorf(y);
    const int x0 = mc::imod_floor((int)fx, d.W), y0 = mc::imod_floor((int)fy, d.H);
    const int x1 = (x0 + 1) % d.W, y1 = (y0 + 1) % d.H;
    const float dx = x - fx, dy = y - fy;
    const float d00 = d.ldep[y0 * d.W + x0], d10 = d.ldep[y0 * d.W + x1];
    const float d01 = d.ldep[y1 * d.W + x0], d11 = d.ldep[y1 * d.W + x1];
    const float s = d.scatter;
    l0.x += s * (-(1.0f - dy) * d00 + (1.0f - dy) * d10 - dy * d01 + dy * d11);
    l0.y += s * (-(1.0f - dx) * d00 - dx * d10 + (1.0f - dx) * d01 + dx * d11);
  }
  const float2 lpv = d.lprev[n];
  d.lpos[n] = make_float2(lpv.x + l0.x, lpv.y + l0.y);
  d.lvel[n] = make_float2((l0.x * d.damp) * d.dt, (l0.y * d.damp) * d.dt);
}

// jp[0]: the step being reversed; jp[1]: the step being taped beside it, the one before
__global__ void k_step_next(AD d) {
  mc::after_previous();
  if (threadIdx.x < 3 && blockIdx.x == 0) d.ntouched[threadIdx.x] = 0;
  if (threadIdx.x < 2 && blockIdx.x == 0) d.jp[threadIdx.x] -= 1;
}

__global__ void k_copy_lpred(AD d) {
  mc::after_previous();
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < d.N) d.lpred0p[n] = d.lpred1[n];
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ host plan
struct mc_grad_plan {
  mc_dims dims{};
  mc_config cfg{};
  float dt = 0.f;
  int T = 0, S = 1, nseg = 0;
  std::vector<int> pairs, bpairs, n_start, n_list, e_start, e_list;
  std::vector<float> ndeg, edeg;
  mc_plan* fwd = nullptr;
  size_t fwd_bytes = 0, total = 0;
  unsigned char* ws = nullptr;
  bool bound = false, have_forward = false, has_act = false;
  long long forwards = 0, backwards = 0;  // calls so far, the present one included (step_graphs)
  // region offsets
  struct R {
    size_t off = 0, bytes = 0;
  };
  R r_fwd, r_pairs, r_bpairs, r_nst, r_nl, r_est, r_el, r_ndeg, r_edeg, r_len, r_kb, r_rst, r_ac, r_aa, r_ao, r_ap,
      r_fdesc;
  bool filter_ready = false;
  R r_wpos, r_wvel, r_wth, r_wra, r_wst, r_wfu, r_wf, r_ck, r_seg, r_segV;
  R r_rest, r_pred0, r_pp, r_tt, r_ibidx, r_ibw, r_sraw, r_stmp, r_uc, r_inv, r_cnt, r_start, r_bucket, r_ovh, r_ovn, r_ovf,
      r_ent, r_touch;
  long long pool = 0;  // where the pool of runs begins in r_ent
  R r_lf0p, r_lv, r_lrho, r_luc, r_lnv, r_lprev, r_lpos, r_lvel, r_lth, r_lp0, r_lp1, r_lt0, r_lt1, r_lcur, r_lthn,
      r_gb, r_racc, r_dc, r_da, r_dp, r_do, r_dr, r_dl, r_dk, r_stv, r_lpred1, r_lpred0p, r_lV, r_ctmp, r_ldep, r_lf0,
      r_lf1;
  size_t state_ck_bytes = 0;  // one checkpoint: pos, vel, theta, f
  AD ad{};
  std::vector<int> c_nstart, c_nodes, c_estart, c_edges, c_bstart, c_bps;  // rod components
  R r_cns, r_cn, r_ces, r_ce, r_cbs, r_cb, r_sargs, r_jp;
  R r_ly, r_lfn, r_lhn;
  std::vector<StepArgs> sargs;
  cudaStream_t cap_stream = nullptr;
  // The recomputation of a segment beside the reverse steps of the one after it (replay_segment)
  bool overlap = false;
  cudaStream_t replay_stream = nullptr;
  cudaEvent_t ev_replayed[2] = {nullptr, nullptr}, ev_reversed[2] = {nullptr, nullptr}, ev_begin = nullptr;
  // Two tapes (tape_step): the second lies tape_bytes behind the first; 0: one
  size_t tape_bytes = 0;
  cudaStream_t tape_stream = nullptr;
  cudaEvent_t ev_tape = nullptr;
  AD tape_ad(int par) const;  // ad with the buffers of tape `par`
  cudaGraphExec_t rev_graphs[6] = {};  // by RevGraph
  int rev_graph_act = -1;              // has_act they were captured with
};

AD mc_grad_plan::tape_ad(int par) const {
  AD d = ad;
  auto shift = [&](auto*& q) { q = reinterpret_cast<std::remove_reference_t<decltype(q)>>((unsigned char*)q + par * tape_bytes); };
  shift(d.rest), shift(d.rest_acc), shift(d.pred0), shift(d.pp), shift(d.tt), shift(d.ib_idx), shift(d.ib_w);
  shift(d.sraw), shift(d.s_tmp), shift(d.uc), shift(d.inv), shift(d.cnt), shift(d.start), shift(d.bucket);
  shift(d.ovf_head), shift(d.ovf_next), shift(d.ovf), shift(d.ent), shift(d.touched), shift(d.ntouched);
  return d;
}

namespace {

thread_local std::string g_gerr;

mc_status gfail(mc_status s, const std::string& m) {
  mc::set_last_error(m.c_str());
  return s;
}

#define GC(call)                                                                                 \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess) return gfail(MC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

size_t al(size_t x) { return (x + 255) / 256 * 256; }

template <typename T>
T* at(unsigned char* ws, const mc_grad_plan::R& r) {
  return reinterpret_cast<T*>(ws + r.off);
}

mc_status copy_state_to(mc_grad_plan* p, float* pos, float* vel, float* th, float* f, const float* spos, const float* svel,
                        const float* sth, const float* sf, cudaStream_t s) {
  const mc_dims& D = p->dims;
  const size_t HW = (size_t)p->ad.lHW;  // f_grid lives on the fluid lattice
  GC(cudaMemcpyAsync(pos, spos, (size_t)D.N * 8, cudaMemcpyDeviceToDevice, s));
  GC(cudaMemcpyAsync(vel, svel, (size_t)D.N * 8, cudaMemcpyDeviceToDevice, s));
  if (D.E) GC(cudaMemcpyAsync(th, sth, (size_t)D.E * 4, cudaMemcpyDeviceToDevice, s));
  GC(cudaMemcpyAsync(f, sf, 9 * HW * 4, cudaMemcpyDeviceToDevice, s));
  return MC_OK;
}

// checkpoint / segment slot layout: pos (2N), vel (2N), theta (E), f (9 lHW), each 256-aligned
struct Slot {
  float *pos, *vel, *th, *f;
};
Slot slot(mc_grad_plan* p, const mc_grad_plan::R& r, int k) {
  const mc_dims& D = p->dims;
  unsigned char* b = p->ws + r.off + (size_t)k * p->state_ck_bytes;
  Slot s;
  s.pos = reinterpret_cast<float*>(b);
  b += al((size_t)D.N * 8);
  s.vel = reinterpret_cast<float*>(b);
  b += al((size_t)D.N * 8);
  s.th = reinterpret_cast<float*>(b);
  b += al((size_t)std::max(D.E, 1) * 4);
  s.f = reinterpret_cast<float*>(b);
  return s;
}

mc_state working_state(mc_grad_plan* p) {
  mc_state w{};
  w.position = at<float>(p->ws, p->r_wpos);
  w.velocity = at<float>(p->ws, p->r_wvel);
  w.theta = at<float>(p->ws, p->r_wth);
  w.rest_lengths = at<float>(p->ws, p->r_len);
  w.bending_rest_angles = at<float>(p->ws, p->r_wra);
  w.bending_stiffness = at<float>(p->ws, p->r_kb);
  w.steric = at<float>(p->ws, p->r_wst);
  w.fluid_velocity = at<float>(p->ws, p->r_wfu);
  w.f_grid = at<float>(p->ws, p->r_wf);
  return w;
}

// Values grouped by key, in the order given: each(put) calls put(key, value) for all of them, the
// same ones each time.
template <class F>
void group_by(int groups, std::vector<int>& start, std::vector<int>& list, F&& each) {
  start.assign(groups + 1, 0);
  each([&](int key, int) { ++start[key + 1]; });
  for (int g = 0; g < groups; ++g) start[g + 1] += start[g];
  list.resize(start[groups]);
  std::vector<int> next(start.begin(), start.end() - 1);
  each([&](int key, int value) { list[next[key]++] = value; });
}

// The first gradient of a short rollout launches its kernels directly: a plan of one gradient would
// spend more on making its graphs (some 0.25 ms each to capture and instantiate, 0.14 to destroy, with
// the GPU idle before the first and after the last) than on launching each kernel (2 us).  48 steps at
// 256^2 13.9 -> 12.9 ms, 12 steps at 640^2 8.6 -> 7.4.  A reverse step has three times the kernels of
// a forward one, so that its graphs pay from fewer steps on.  First pass of a plan in us, launched
// directly and by graphs: forward of 48 and 64 steps at 256^2 4,397 and 4,717, 5,792 and 6,173, at
// 640^2 5,321 and 5,500, 6,947 and 7,014 (of 96 at 256^2, always by graphs, 8,923); reverse of 16 steps
// of a 64^2 lattice 2,872 and 2,920, at 256^2 2,806 and 2,946, of 48 there 7,210 and 7,146.
// A plan that is kept makes its graphs at the second gradient, since each further one is then faster:
// forward of 48 steps at 640^2 5,279 -> 4,998, reverse of 16 steps of a 64^2 lattice 2,837 -> 2,346.
int step_graphs(const mc_grad_plan* p) { return p->T > kDirectSteps || p->forwards > 1; }
bool reverse_graphs(const mc_grad_plan* p) { return p->T > kDirectReverse || p->backwards > 1; }

// Open a rollout of the forward plan on the working state, actuated from step t0 (the
// static rest angles restored first when there is no actuation).
mc_status begin_fwd(mc_grad_plan* p, int t0, cudaStream_t s) {
  mc_state w = working_state(p);
  mc_actuation a{};
  const mc_actuation* ap = nullptr;
  if (p->has_act) {
    a.c = at<float>(p->ws, p->r_ac);
    a.amp = at<float>(p->ws, p->r_aa);
    a.omega = at<float>(p->ws, p->r_ao);
    a.phase = at<float>(p->ws, p->r_ap);
    a.t0 = t0;
    ap = &a;
  } else if (p->dims.B) {
    GC(cudaMemcpyAsync(w.bending_rest_angles, at<float>(p->ws, p->r_rst), (size_t)p->dims.B * 4,
                       cudaMemcpyDeviceToDevice, s));
  }
  const mc_actuation* const acts[1] = {ap};
  return mc_rollout_begin(p->fwd, &w, acts, nullptr, s);
}

// Where the inputs of step j of segment k are kept: neighbouring segments apart when they overlap.
int segment_slot(const mc_grad_plan* p, int k, int j) { return (p->overlap && (k & 1) ? p->S : 0) + j; }

// The step inputs of segment k from its checkpoint: one rollout over the segment, the populations
// of every step's input snapshot from the open rollout (no per-step entry/exit conversion).
mc_status replay_segment(mc_grad_plan* p, int k, cudaStream_t s) {
  const mc_dims& D = p->dims;
  const size_t HW = (size_t)D.H * D.W, LHW = (size_t)p->ad.lHW;
  unsigned char* w = p->ws;
  const int t0 = k * p->S, len = std::min(p->S, p->T - t0);
  Slot ck = slot(p, p->r_ck, k);
  mc_status st = copy_state_to(p, at<float>(w, p->r_wpos), at<float>(w, p->r_wvel), at<float>(w, p->r_wth),
                               at<float>(w, p->r_wf), ck.pos, ck.vel, ck.th, ck.f, s);
  if (st != MC_OK) return st;
  st = begin_fwd(p, t0, s);
  if (st != MC_OK) return st;
  for (int j = 0; j < len; ++j) {
    const int at_j = segment_slot(p, k, j);
    Slot sj = slot(p, p->r_seg, at_j);
    GC(cudaMemcpyAsync(sj.pos, at<float>(w, p->r_wpos), (size_t)D.N * 8, cudaMemcpyDeviceToDevice, s));
    GC(cudaMemcpyAsync(sj.vel, at<float>(w, p->r_wvel), (size_t)D.N * 8, cudaMemcpyDeviceToDevice, s));
    if (D.E) GC(cudaMemcpyAsync(sj.th, at<float>(w, p->r_wth), (size_t)D.E * 4, cudaMemcpyDeviceToDevice, s));
    if (p->ad.fluid) {
      st = mc::rollout_snapshot_f(p->fwd, sj.f, s);
      if (st != MC_OK) return st;
    } else {
      GC(cudaMemcpyAsync(sj.f, at<float>(w, p->r_wf), 9 * LHW * 4, cudaMemcpyDeviceToDevice, s));
    }
    st = mc_rollout_advance(p->fwd, 1, step_graphs(p), 1, s);
    if (st != MC_OK) return st;
    GC(cudaMemcpyAsync(w + p->r_segV.off + (size_t)at_j * al(HW * 4), w + p->r_wst.off, HW * 4,
                       cudaMemcpyDeviceToDevice, s));
  }
  return mc_rollout_end(p->fwd, s);
}

mc_status run_fwd(mc_grad_plan* p, int steps, int t0, cudaStream_t s) {
  mc_state w = working_state(p);
  mc_actuation a{};
  const mc_actuation* ap = nullptr;
  if (p->has_act) {
    a.c = at<float>(p->ws, p->r_ac);
    a.amp = at<float>(p->ws, p->r_aa);
    a.omega = at<float>(p->ws, p->r_ao);
    a.phase = at<float>(p->ws, p->r_ap);
    a.t0 = t0;
    ap = &a;
  } else if (p->dims.B) {
    // the static rest angles (the actuation, when used, overwrites this copy)
    GC(cudaMemcpyAsync(w.bending_rest_angles, at<float>(p->ws, p->r_rst), (size_t)p->dims.B * 4,
                       cudaMemcpyDeviceToDevice, s));
  }
  const mc_actuation* const acts[1] = {ap};
  return mc_rollout(p->fwd, &w, steps, acts, nullptr, step_graphs(p), s);
}

// Enqueues kernels, each chained to the one before on its stream.
struct Chain {
  cudaStream_t s;
  bool behind = false;  // the stream's last operation here is a kernel
  template <class... P, class... A>
  void operator()(void (*kernel)(P...), int grid, int threads, A... args) {
    mc::Launch l{nullptr, nullptr, 0, grid, s, behind};
    mc::launch(l, kernel, threads, 0, args...);
    behind = true;
  }
};

// The forward side of a step, kept for its reverse; its inputs come from sa[*jp].
void tape_step(const AD& d, cudaStream_t s) {
  const int TB = 256;
  Chain go{s};
  go(k_rest, nblk(std::max(d.B, 1), TB), TB, d);
  go(k_pred, nblk(std::max(4LL * d.N, (long long)d.E), 128), 128, d);
  go(d.solver == MC_SOLVER_COSSERAT ? k_cos_fwd : k_pbd_fwd, d.ncomp, kPbdThreads, d);
  if (!d.fluid) return;
  if (d.K <= 4)
    go(k_ib_weights4, nblk(4LL * d.NI, 128), 128, d);
  else
    go(k_ib_weights, nblk(d.NI, TB), TB, d);
  const int most = std::min((long long)d.NI * d.KK, (long long)d.lHW);  // touched cells at most
  go(k_cell_order, nblk(most, 128), 128, d);
  go(k_macro, nblk(d.lHW, TB), TB, d);
  for (int it = 0; it < d.iters; ++it) {
    go(k_ib_interp, nblk(d.NI, kPointThreads), kPointThreads, d, it);
    go(k_ib_spread, nblk(most, 128), 128, d);
  }
}

// The reverse of a taped step, up to k_step_next.
void reverse_step(mc_grad_plan* p, const AD& d, cudaStream_t s) {
  const int TB = 256;
  const int nNE = std::max(d.N, d.E);
  if (d.fluid && d.iters == 0) cudaMemsetAsync(d.lnv, 0, (size_t)d.NI * 8, s);
  if (d.steric) cudaMemsetAsync(d.lV, 0, (size_t)d.HW * 4, s);
  Chain go{s};
  if (d.fluid) {
    const int most = std::min((long long)d.NI * d.KK, (long long)d.lHW);
    go(k_lbm_adj1, nblk(d.lHW, TB), TB, d);
    for (int it = d.iters - 1; it >= 0; --it) {
      go(k_ib_rev_node, nblk(d.NI, kPointThreads), kPointThreads, d, it);
      go(k_ib_rev_cell, nblk(most, 128), 128, d);
    }
    go(k_lbm_adj2, nblk(d.lHW, TB), TB, d);
  }
  go(k_node_adj, nblk(nNE, TB), TB, d);
  go(d.solver == MC_SOLVER_COSSERAT ? k_cos_rev : k_pbd_rev, d.ncomp, kPbdThreads, d);
  if (d.steric) {
    const int most = std::min(16LL * d.N, (long long)d.HW);
    go(k_steric_adj_node, nblk(4LL * d.N, 128), 128, d);
    go(k_cell_order, nblk(most, 128), 128, d);
    go(k_gather_field, nblk(most, TB), TB, d, (const float*)d.st_val, d.lV);
    // the spectral filter is real and even, so it is its own adjoint: the forward plan's
    // filter kernels map the sample cotangent lV to the deposit cotangent ldep
    mc::filter_launch(p->fwd, p->ws + p->r_fdesc.off, s);
  } else {
    go(k_copy_lpred, nblk(d.N, TB), TB, d);
  }
  go(k_steric_adj_cic, nblk(d.N, TB), TB, d);
}

// What a segment's reverse is made of, graphs or direct launches.  With two tapes (steps of odd and even number), the
// tape of step j - 1 runs beside the reverse of step j: neither fills more than a few SMs.
enum RevGraph { kTapeEven, kTapeOdd, kBothEven, kBothOdd, kReverseEven, kWhole };

void enqueue_reverse(mc_grad_plan* p, int which, cudaStream_t s) {
  const int par = which & 1;
  AD d = p->ad;
  if (which == kWhole) {
    tape_step(d, s);
    reverse_step(p, d, s);
    mc::launch(mc::Launch{nullptr, nullptr, 0, 1, s, true}, k_step_next, 32, 0, d);
    return;
  }
  d = p->tape_ad(par);
  if (which == kTapeEven || which == kTapeOdd) return tape_step(d, s);
  const bool both = which != kReverseEven;
  if (both) {
    AD t = p->tape_ad(par ^ 1);
    t.jp = d.jp + 1;
    cudaEventRecord(p->ev_tape, s);
    cudaStreamWaitEvent(p->tape_stream, p->ev_tape, 0);
    tape_step(t, p->tape_stream);
  }
  reverse_step(p, d, s);
  if (both) {
    cudaEventRecord(p->ev_tape, p->tape_stream);
    cudaStreamWaitEvent(s, p->ev_tape, 0);
  }
  mc::launch(mc::Launch{nullptr, nullptr, 0, 1, s, !both}, k_step_next, 32, 0, d);
}

// The captured graph `which`, made on first use.
mc_status rev_graph(mc_grad_plan* p, int which, cudaGraphExec_t* out) {
  cudaGraphExec_t& x = p->rev_graphs[which];
  if (!x) {
    cudaGraph_t g;
    GC(cudaStreamBeginCapture(p->cap_stream, cudaStreamCaptureModeThreadLocal));
    enqueue_reverse(p, which, p->cap_stream);
    cudaError_t e = cudaStreamEndCapture(p->cap_stream, &g);
    if (e != cudaSuccess) return gfail(MC_ERR_CUDA, std::string("capture of the reverse step: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&x, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      x = nullptr;
      return gfail(MC_ERR_CUDA, std::string("instantiating the reverse step: ") + cudaGetErrorString(e));
    }
  }
  *out = x;
  return MC_OK;
}

void drop_rev_graphs(mc_grad_plan* p) {
  for (cudaGraphExec_t& x : p->rev_graphs) {
    if (x) cudaGraphExecDestroy(x);
    x = nullptr;
  }
}

}  // namespace

extern "C" {

mc_status mc_grad_plan_create(const mc_dims* dims, const mc_config* cfg, float dt, const int32_t* pairs,
                              const int32_t* bending_pairs, int32_t num_steps, int32_t checkpoint_every,
                              mc_grad_plan** out) {
  mc::set_last_error("");
  if (!dims || !cfg || !out) return gfail(MC_ERR_INVALID, "null argument");
  *out = nullptr;
  const mc_dims D = *dims;
  if (D.N < 1 || D.E < 0 || D.B < 0 || D.H < 4 || D.W < 4) return gfail(MC_ERR_INVALID, "bad dims");
  if ((D.E && !pairs) || (D.B && !bending_pairs)) return gfail(MC_ERR_INVALID, "null topology");
  if (num_steps < 0) return gfail(MC_ERR_INVALID, "negative num_steps");
  if ((long long)D.H * D.W > kMaxCells) return gfail(MC_ERR_UNSUPPORTED, "grid too large for the gradient path");
  if (cfg->ibm_kernel_size < 1 || cfg->ibm_kernel_size * cfg->ibm_kernel_size > kMaxKK)
    return gfail(MC_ERR_UNSUPPORTED, "ibm_kernel_size outside 1..8");
  if (cfg->synthetic_node_width < 0.0f) return gfail(MC_ERR_INVALID, "synthetic_node_width must be >= 0");
  if ((D.fluid_H > 0) != (D.fluid_W > 0) || D.fluid_H < 0 || D.fluid_W < 0)
    return gfail(MC_ERR_INVALID, "fluid_H and fluid_W must both be 0 (the domain grid) or both > 0");
  if ((long long)std::max(D.fluid_H, 0) * std::max(D.fluid_W, 0) > kMaxCells)
    return gfail(MC_ERR_UNSUPPORTED, "fluid lattice too large for the gradient path");
  if (cfg->solver_type != MC_SOLVER_PBD && cfg->solver_type != MC_SOLVER_COSSERAT)
    return gfail(MC_ERR_INVALID, "solver_type must be MC_SOLVER_PBD or MC_SOLVER_COSSERAT");
  if (cfg->solver_type == MC_SOLVER_COSSERAT && !(cfg->solver_dt > 0.0))
    return gfail(MC_ERR_INVALID, "the stable-Cosserat solver needs solver_dt > 0");
  mc_grad_plan* p = new mc_grad_plan();
  p->dims = D;
  p->cfg = *cfg;
  p->dt = dt;
  p->T = num_steps;
  int S = checkpoint_every;
  if (S <= 0) S = std::max(1, (int)std::ceil(std::sqrt((double)std::max(num_steps, 1))));
  p->S = S;
  p->nseg = (num_steps + S - 1) / S;
  p->pairs.assign(pairs, pairs + 2 * (size_t)D.E);
  p->bpairs.assign(bending_pairs, bending_pairs + 2 * (size_t)D.B);
  for (int e = 0; e < D.E; ++e)
    for (int j = 0; j < 2; ++j)
      if (p->pairs[2 * e + j] < 0 || p->pairs[2 * e + j] >= D.N) {
        delete p;
        return gfail(MC_ERR_INVALID, "pairs index out of range");
      }
  for (int b = 0; b < D.B; ++b)
    for (int j = 0; j < 2; ++j)
      if (p->bpairs[2 * b + j] < 0 || p->bpairs[2 * b + j] >= D.E) {
        delete p;
        return gfail(MC_ERR_INVALID, "bending_pairs index out of range");
      }
  // gather lists in scatter order: sources first (in edge order), then targets
  auto ends = [](const std::vector<int>& ab, int count) {
    return [&ab, count](auto&& put) {
      for (int q = 0; q < 2; ++q)
        for (int i = 0; i < count; ++i) put(ab[2 * i + q], i * 2 + q);
    };
  };
  group_by(D.N, p->n_start, p->n_list, ends(p->pairs, D.E));
  p->ndeg.resize(D.N);
  for (int n = 0; n < D.N; ++n) p->ndeg[n] = std::max((float)(p->n_start[n + 1] - p->n_start[n]), 1.0f);
  group_by(D.E, p->e_start, p->e_list, ends(p->bpairs, D.B));
  p->edeg.resize(D.E);
  for (int e = 0; e < D.E; ++e) p->edeg[e] = std::max((float)(p->e_start[e + 1] - p->e_start[e]), 1.0f);
  {
    // rod components: union-find over the edges; members listed in ascending order
    std::vector<int> par(D.N);
    for (int n = 0; n < D.N; ++n) par[n] = n;
    auto find = [&](int x) {
      while (par[x] != x) {
        par[x] = par[par[x]];
        x = par[x];
      }
      return x;
    };
    for (int e = 0; e < D.E; ++e) {
      const int a = find(p->pairs[2 * e]), b = find(p->pairs[2 * e + 1]);
      if (a != b) par[std::max(a, b)] = std::min(a, b);
    }
    std::vector<int> cid(D.N, -1);
    int nc = 0;
    for (int n = 0; n < D.N; ++n) {
      const int r = find(n);
      if (cid[r] < 0) cid[r] = nc++;
      cid[n] = cid[r];
    }
    group_by(nc, p->c_nstart, p->c_nodes, [&](auto&& put) {
      for (int n = 0; n < D.N; ++n) put(cid[n], n);
    });
    group_by(nc, p->c_estart, p->c_edges, [&](auto&& put) {
      for (int e = 0; e < D.E; ++e) put(cid[p->pairs[2 * e]], e);
    });
    group_by(nc, p->c_bstart, p->c_bps, [&](auto&& put) {
      for (int b = 0; b < D.B; ++b) put(cid[p->pairs[2 * p->bpairs[2 * b]]], b);
    });
  }
  // forward plan (same kernels as mc_rollout)
  const int32_t* pp[1] = {pairs};
  const int32_t* bb[1] = {bending_pairs};
  mc_status st = mc_plan_create(1, &D, cfg, &dt, pp, bb, &p->fwd);
  if (st != MC_OK) {
    delete p;
    return st;
  }
  p->fwd_bytes = mc_plan_workspace_bytes(p->fwd);
  // layout
  const size_t N = D.N, E = std::max(D.E, 1), B = std::max(D.B, 1), HW = (size_t)D.H * D.W;
  const size_t LHW = D.fluid_H > 0 ? (size_t)D.fluid_H * D.fluid_W : HW;  // fluid lattice cells
  const size_t CHW = std::max(HW, LHW);                                    // CSR cells
  const size_t NI = N * (cfg->enable_fluid && cfg->synthetic_node_width > 0.0f ? 2 : 1);  // IB points
  const int C = cfg->cycles_per_step, KK = cfg->ibm_kernel_size * cfg->ibm_kernel_size;
  const int iters = std::max(cfg->ibm_iterations, 1);
  size_t o = 0;
  auto take = [&](mc_grad_plan::R& r, size_t bytes) {
    r.off = o;
    r.bytes = bytes;
    o += al(std::max<size_t>(bytes, 4));
  };
  take(p->r_fwd, p->fwd_bytes);
  take(p->r_pairs, E * 8);
  take(p->r_bpairs, B * 8);
  take(p->r_nst, (N + 1) * 4);
  take(p->r_nl, std::max<size_t>(p->n_list.size(), 1) * 4);
  take(p->r_est, (E + 1) * 4);
  take(p->r_el, std::max<size_t>(p->e_list.size(), 1) * 4);
  take(p->r_ndeg, N * 4);
  take(p->r_edeg, E * 4);
  take(p->r_len, E * 4);
  take(p->r_kb, B * 4);
  take(p->r_rst, B * 4);
  take(p->r_ac, B * 4);
  take(p->r_aa, B * 4);
  take(p->r_ao, B * 4);
  take(p->r_ap, B * 4);
  take(p->r_wpos, N * 8);
  take(p->r_wvel, N * 8);
  take(p->r_wth, E * 4);
  take(p->r_wra, B * 4);
  take(p->r_wst, HW * 4);
  take(p->r_wfu, 2 * LHW * 4);
  take(p->r_wf, 9 * LHW * 4);
  p->state_ck_bytes = al(N * 8) * 2 + al(E * 4) + al(9 * LHW * 4);
  take(p->r_ck, std::max(p->nseg, 1) * p->state_ck_bytes);
  // a second copy of the segment's inputs, unless it is of a size that a user would notice
  const size_t seg_bytes = (size_t)S * (p->state_ck_bytes + al(HW * 4));
  p->overlap = p->nseg > 1 && seg_bytes <= kOverlapBytes;
  const size_t copies = p->overlap ? 2 : 1;
  take(p->r_seg, copies * S * p->state_ck_bytes);
  take(p->r_segV, copies * S * al(HW * 4));
  take(p->r_rest, B * 4);
  take(p->r_pred0, N * 8);
  take(p->r_pp, (size_t)(C + 1) * N * 8);
  take(p->r_tt, (size_t)(C + 1) * E * 4);
  take(p->r_ibidx, NI * KK * 4);
  take(p->r_ibw, NI * KK * 4);
  take(p->r_sraw, (size_t)iters * NI * 8);
  take(p->r_stmp, NI * 8);
  take(p->r_uc, 2 * LHW * 4);
  take(p->r_inv, LHW * 4);
  const size_t entries = std::max<size_t>(NI * KK, 16 * N);
  const size_t rows = std::min(entries, CHW);
  p->pool = (long long)(rows * kCellBucket);
  take(p->r_cnt, CHW * 4);
  take(p->r_bucket, CHW * kCellBucket * 4);
  take(p->r_ovh, CHW * 4);
  take(p->r_ovn, entries * 4);
  take(p->r_ovf, entries * 4);
  take(p->r_start, CHW * 4);
  take(p->r_ent, (rows * kCellBucket + 2 * entries) * 4);
  take(p->r_touch, rows * 4 + 256);
  take(p->r_racc, B * 4);
  p->tape_bytes = 0;
  if (S > 1 && num_steps > 1 && o - p->r_rest.off <= kOverlapBytes) {
    p->tape_bytes = o - p->r_rest.off;
    o += p->tape_bytes;
  }
  take(p->r_lf0p, 9 * LHW * 4);
  take(p->r_lv, 2 * LHW * 4);
  take(p->r_lrho, LHW * 4);
  take(p->r_luc, 2 * LHW * 4);
  take(p->r_lnv, NI * 8);
  take(p->r_lprev, N * 8);
  take(p->r_lpos, N * 8);
  take(p->r_lvel, N * 8);
  take(p->r_lth, E * 4);
  take(p->r_lp0, N * 8);
  take(p->r_lp1, N * 8);
  take(p->r_lt0, E * 4);
  take(p->r_lt1, E * 4);
  take(p->r_lcur, E * 8);
  take(p->r_lthn, E * 4);
  take(p->r_gb, B * 4);
  take(p->r_ly, N * 8);
  take(p->r_lfn, N * 8);
  take(p->r_lhn, N * 4);
  take(p->r_dc, B * 4);
  take(p->r_da, B * 4);
  take(p->r_dp, B * 4);
  take(p->r_do, B * 4);
  take(p->r_dr, B * 4);
  take(p->r_dl, E * 4);
  take(p->r_dk, B * 4);
  take(p->r_stv, 16 * N * 4);
  take(p->r_lpred1, N * 8);
  take(p->r_lpred0p, N * 8);
  take(p->r_lV, HW * 4);
  take(p->r_ctmp, HW * 4);
  take(p->r_ldep, HW * 4);
  take(p->r_lf0, 9 * LHW * 4);
  take(p->r_lf1, 9 * LHW * 4);
  take(p->r_cns, p->c_nstart.size() * 4);
  take(p->r_cn, std::max<size_t>(p->c_nodes.size(), 1) * 4);
  take(p->r_ces, p->c_estart.size() * 4);
  take(p->r_ce, std::max<size_t>(p->c_edges.size(), 1) * 4);
  take(p->r_cbs, p->c_bstart.size() * 4);
  take(p->r_cb, std::max<size_t>(p->c_bps.size(), 1) * 4);
  take(p->r_sargs, (size_t)S * sizeof(StepArgs));
  take(p->r_fdesc, mc::filter_desc_bytes());
  take(p->r_jp, 8);
  p->total = o;
  *out = p;
  return MC_OK;
}

void mc_grad_plan_destroy(mc_grad_plan* p) {
  if (!p) return;
  drop_rev_graphs(p);
  if (p->tape_stream) cudaStreamDestroy(p->tape_stream);
  if (p->ev_tape) cudaEventDestroy(p->ev_tape);
  if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
  if (p->replay_stream) cudaStreamDestroy(p->replay_stream);
  for (cudaEvent_t e : {p->ev_replayed[0], p->ev_replayed[1], p->ev_reversed[0], p->ev_reversed[1], p->ev_begin})
    if (e) cudaEventDestroy(e);
  if (p->fwd) mc_plan_destroy(p->fwd);
  delete p;
}

size_t mc_grad_plan_workspace_bytes(const mc_grad_plan* p) { return p ? p->total : 0; }

int32_t mc_grad_plan_checkpoint_every(const mc_grad_plan* p) { return p ? p->S : 0; }

mc_status mc_grad_plan_bind(mc_grad_plan* p, void* workspace, size_t bytes, void* stream) {
  mc::set_last_error("");
  if (!p) return gfail(MC_ERR_INVALID, "null plan");
  if (!workspace || bytes < p->total || ((uintptr_t)workspace & 255))
    return gfail(MC_ERR_WORKSPACE, "workspace missing, too small or not 256-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  p->ws = (unsigned char*)workspace;
  mc_status st = mc_plan_bind(p->fwd, p->ws + p->r_fwd.off, p->fwd_bytes, stream);
  if (st != MC_OK) return st;
  std::vector<mc::Upload> ups;
  auto up = [&](const mc_grad_plan::R& r, const void* src, size_t n) -> cudaError_t {
    if (n) ups.push_back({p->ws + r.off, src, n});
    return cudaSuccess;
  };
  GC(up(p->r_pairs, p->pairs.data(), p->pairs.size() * 4));
  GC(up(p->r_bpairs, p->bpairs.data(), p->bpairs.size() * 4));
  GC(up(p->r_nst, p->n_start.data(), p->n_start.size() * 4));
  GC(up(p->r_nl, p->n_list.data(), p->n_list.size() * 4));
  GC(up(p->r_est, p->e_start.data(), p->e_start.size() * 4));
  GC(up(p->r_el, p->e_list.data(), p->e_list.size() * 4));
  GC(up(p->r_ndeg, p->ndeg.data(), p->ndeg.size() * 4));
  GC(up(p->r_edeg, p->edeg.data(), p->edeg.size() * 4));
  GC(up(p->r_cns, p->c_nstart.data(), p->c_nstart.size() * 4));
  GC(up(p->r_cn, p->c_nodes.data(), p->c_nodes.size() * 4));
  GC(up(p->r_ces, p->c_estart.data(), p->c_estart.size() * 4));
  GC(up(p->r_ce, p->c_edges.data(), p->c_edges.size() * 4));
  GC(up(p->r_cbs, p->c_bstart.data(), p->c_bstart.size() * 4));
  GC(up(p->r_cb, p->c_bps.data(), p->c_bps.size() * 4));
  GC(mc::stage_uploads(ups.data(), (int)ups.size(), s));
  drop_rev_graphs(p);
  p->filter_ready = false;
  if (!p->cap_stream) GC(cudaStreamCreateWithFlags(&p->cap_stream, cudaStreamNonBlocking));
  if (p->overlap) {
    if (!p->replay_stream) GC(cudaStreamCreateWithFlags(&p->replay_stream, cudaStreamNonBlocking));
    for (cudaEvent_t* e : {&p->ev_replayed[0], &p->ev_replayed[1], &p->ev_reversed[0], &p->ev_reversed[1], &p->ev_begin})
      if (!*e) GC(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  if (p->tape_bytes) {
    if (!p->tape_stream) GC(cudaStreamCreateWithFlags(&p->tape_stream, cudaStreamNonBlocking));
    if (!p->ev_tape) GC(cudaEventCreateWithFlags(&p->ev_tape, cudaEventDisableTiming));
  }
  for (int c = 0; c < (p->tape_bytes ? 2 : 1); ++c) {
    unsigned char* at_c = p->ws + c * p->tape_bytes;
    GC(cudaMemsetAsync(at_c + p->r_cnt.off, 0, p->r_cnt.bytes, s));
    GC(cudaMemsetAsync(at_c + p->r_ovh.off, 0xff, p->r_ovh.bytes, s));
    GC(cudaMemsetAsync(at_c + p->r_touch.off, 0, 256, s));
  }
  const mc_config& c = p->cfg;
  const mc_dims& D = p->dims;
  AD& d = p->ad;
  d = AD{};
  d.H = D.H;
  d.W = D.W;
  d.N = D.N;
  d.E = D.E;
  d.B = D.B;
  d.HW = D.H * D.W;
  d.lH = D.fluid_H > 0 ? D.fluid_H : D.H;
  d.lW = D.fluid_W > 0 ? D.fluid_W : D.W;
  d.lHW = d.lH * d.lW;
  d.C = c.cycles_per_step;
  d.iters = c.ibm_iterations;
  d.K = c.ibm_kernel_size;
  d.KK = d.K * d.K;
  d.steric = c.enable_steric;
  d.fluid = c.enable_fluid;
  d.nskip = c.steric_neighbor_skip;
  d.dt = p->dt;
  d.damp = c.damping;
  d.st_strength = c.steric_strength;
  d.sigma = c.steric_sigma;
  d.scatter = c.steric_scatter_value;
  d.kstretch = c.stiffness_stretch;
  d.kshear = c.stiffness_shear;
  d.solver = c.solver_type;
  d.force_clamp = c.enable_force_clamp;
  d.NI = D.N * (c.enable_fluid && c.synthetic_node_width > 0.0f ? 2 : 1);
  d.syn_w = c.synthetic_node_width;
  // scale = (lW / H, lH / W): the reference's axis order (fluid.py:222-226)
  const double sxd = (double)d.lW / (double)D.H, syd = (double)d.lH / (double)D.W;
  d.syn_ms = (float)(0.5 * (sxd + syd));
  d.cos_w = c.solver_type == MC_SOLVER_COSSERAT ? (float)(1.0 / (c.solver_dt * c.solver_dt)) : 0.0f;
  const float scx = (float)sxd, scy = (float)syd;
  d.scx = scx;
  d.scy = scy;
  d.vmax = (float)((double)c.max_fluid_velocity * (0.5 * (sxd + syd)));
  d.relax = c.ibm_relaxation;
  d.mass = c.node_mass;
  {
    // omega+ = clip(1/(3 nu + 0.5), 0, 1.9); omega- from the magic parameter (fluid.py:155-161)
    const float wp = std::min(std::max((float)(1.0 / (3.0 * c.viscosity + 0.5)), 0.0f), 1.9f);
    const float eps = 1.1920928955078125e-07f;
    const float off = 1.0f / std::max(wp, eps) - 0.5f;
    const float wm = 1.0f / (c.lambda_trt / std::max(off, eps) + 0.5f);
    d.wp = wp;
    d.wm = wm;
    d.cp = 1.0f - 0.5f * wp;
    d.cm = 1.0f - 0.5f * wm;
  }
  d.sdtx = scx * p->dt;
  d.sdty = scy * p->dt;
  unsigned char* w = p->ws;
  d.pairs = at<int2>(w, p->r_pairs);
  d.bpairs = at<int2>(w, p->r_bpairs);
  d.n_start = at<int>(w, p->r_nst);
  d.n_list = at<int>(w, p->r_nl);
  d.e_start = at<int>(w, p->r_est);
  d.e_list = at<int>(w, p->r_el);
  d.ndeg = at<float>(w, p->r_ndeg);
  d.edeg = at<float>(w, p->r_edeg);
  d.rest_len = at<float>(w, p->r_len);
  d.kb = at<float>(w, p->r_kb);
  d.rest_static = at<float>(w, p->r_rst);
  d.act_c = at<float>(w, p->r_ac);
  d.act_amp = at<float>(w, p->r_aa);
  d.act_om = at<float>(w, p->r_ao);
  d.act_ph = at<float>(w, p->r_ap);
  d.rest = at<float>(w, p->r_rest);
  d.pred0 = at<float2>(w, p->r_pred0);
  d.pp = at<float2>(w, p->r_pp);
  d.tt = at<float>(w, p->r_tt);
  d.ib_idx = at<int>(w, p->r_ibidx);
  d.ib_w = at<float>(w, p->r_ibw);
  d.sraw = at<float2>(w, p->r_sraw);
  d.s_tmp = at<float2>(w, p->r_stmp);
  d.uc = at<float2>(w, p->r_uc);
  d.inv = at<float>(w, p->r_inv);
  d.cnt = at<int>(w, p->r_cnt);
  d.start = at<int>(w, p->r_start);
  d.bucket = at<int>(w, p->r_bucket);
  d.ovf_head = at<int>(w, p->r_ovh);
  d.ovf_next = at<int>(w, p->r_ovn);
  d.ovf = at<int>(w, p->r_ovf);
  d.pool = (int)p->pool;
  d.ent = at<int>(w, p->r_ent);
  d.ntouched = at<int>(w, p->r_touch);
  d.touched = d.ntouched + 64;
  d.lf0p = at<float>(w, p->r_lf0p);
  d.lv = at<float>(w, p->r_lv);
  d.lrho = at<float>(w, p->r_lrho);
  d.luc = at<float2>(w, p->r_luc);
  d.lnv = at<float2>(w, p->r_lnv);
  d.lprev = at<float2>(w, p->r_lprev);
  d.lpos = at<float2>(w, p->r_lpos);
  d.lvel = at<float2>(w, p->r_lvel);
  d.lth = at<float>(w, p->r_lth);
  d.lp[0] = at<float2>(w, p->r_lp0);
  d.lp[1] = at<float2>(w, p->r_lp1);
  d.lt[0] = at<float>(w, p->r_lt0);
  d.lt[1] = at<float>(w, p->r_lt1);
  d.lcur = at<float2>(w, p->r_lcur);
  d.lthn = at<float>(w, p->r_lthn);
  d.gb = at<float>(w, p->r_gb);
  d.ly = at<float2>(w, p->r_ly);
  d.lfn = at<float2>(w, p->r_lfn);
  d.lhn = at<float>(w, p->r_lhn);
  d.rest_acc = at<float>(w, p->r_racc);
  d.d_c = at<float>(w, p->r_dc);
  d.d_amp = at<float>(w, p->r_da);
  d.d_ph = at<float>(w, p->r_dp);
  d.d_om = at<float>(w, p->r_do);
  d.d_rest = at<float>(w, p->r_dr);
  d.d_len = at<float>(w, p->r_dl);
  d.d_kb = at<float>(w, p->r_dk);
  d.st_val = at<float>(w, p->r_stv);
  d.lpred1 = at<float2>(w, p->r_lpred1);
  d.lpred0p = at<float2>(w, p->r_lpred0p);
  d.lV = at<float>(w, p->r_lV);
  d.ctmp = at<float>(w, p->r_ctmp);
  d.ldep = at<float>(w, p->r_ldep);
  d.ncomp = (int)p->c_nstart.size() - 1;
  d.c_nstart = at<int>(w, p->r_cns);
  d.c_nodes = at<int>(w, p->r_cn);
  d.c_estart = at<int>(w, p->r_ces);
  d.c_edges = at<int>(w, p->r_ce);
  d.c_bstart = at<int>(w, p->r_cbs);
  d.c_bps = at<int>(w, p->r_cb);
  d.sa = at<StepArgs>(w, p->r_sargs);
  d.jp = at<int>(w, p->r_jp);
  p->bound = true;
  return MC_OK;
}

mc_status mc_grad_forward(mc_grad_plan* p, const mc_state* state, const mc_actuation* act, void* stream) {
  mc::set_last_error("");
  if (!p || !state) return gfail(MC_ERR_INVALID, "null argument");
  if (!p->bound) return gfail(MC_ERR_NOT_BOUND, "mc_grad_plan_bind() was not called");
  cudaStream_t s = (cudaStream_t)stream;
  const mc_dims& D = p->dims;
  const size_t HW = (size_t)D.H * D.W;
  const size_t LHW = (size_t)p->ad.lHW;  // fluid lattice cells
  unsigned char* w = p->ws;
  auto cp = [&](const mc_grad_plan::R& r, const void* src, size_t n) -> cudaError_t {
    if (n == 0 || !src) return cudaSuccess;
    return cudaMemcpyAsync(w + r.off, src, n, cudaMemcpyDeviceToDevice, s);
  };
  if (!state->position || !state->velocity || !state->f_grid || (D.E && (!state->theta || !state->rest_lengths)) ||
      (D.B && (!state->bending_rest_angles || !state->bending_stiffness)))
    return gfail(MC_ERR_INVALID, "null state array");
  GC(cp(p->r_wpos, state->position, (size_t)D.N * 8));
  GC(cp(p->r_wvel, state->velocity, (size_t)D.N * 8));
  GC(cp(p->r_wth, state->theta, (size_t)D.E * 4));
  GC(cp(p->r_len, state->rest_lengths, (size_t)D.E * 4));
  GC(cp(p->r_kb, state->bending_stiffness, (size_t)D.B * 4));
  GC(cp(p->r_rst, state->bending_rest_angles, (size_t)D.B * 4));
  GC(cp(p->r_wra, state->bending_rest_angles, (size_t)D.B * 4));
  if (state->steric) GC(cp(p->r_wst, state->steric, HW * 4));
  else GC(cudaMemsetAsync(w + p->r_wst.off, 0, HW * 4, s));
  if (state->fluid_velocity) GC(cp(p->r_wfu, state->fluid_velocity, 2 * LHW * 4));
  else GC(cudaMemsetAsync(w + p->r_wfu.off, 0, 2 * LHW * 4, s));
  GC(cp(p->r_wf, state->f_grid, 9 * LHW * 4));
  p->has_act = act != nullptr;
  if (act) {
    if (D.B && (!act->c || !act->amp || !act->omega || !act->phase)) return gfail(MC_ERR_INVALID, "null actuation array");
    if (act->t0 != 0) return gfail(MC_ERR_UNSUPPORTED, "the gradient path starts its actuation clock at t0 = 0");
    GC(cp(p->r_ac, act->c, (size_t)D.B * 4));
    GC(cp(p->r_aa, act->amp, (size_t)D.B * 4));
    GC(cp(p->r_ao, act->omega, (size_t)D.B * 4));
    GC(cp(p->r_ap, act->phase, (size_t)D.B * 4));
  }
  p->ad.has_act = p->has_act ? 1 : 0;
  ++p->forwards;
  for (int k = 0; k < p->nseg; ++k) {
    Slot ck = slot(p, p->r_ck, k);
    mc_status st = copy_state_to(p, ck.pos, ck.vel, ck.th, ck.f, at<float>(w, p->r_wpos), at<float>(w, p->r_wvel),
                                 at<float>(w, p->r_wth), at<float>(w, p->r_wf), s);
    if (st != MC_OK) return st;
    const int len = std::min(p->S, p->T - k * p->S);
    st = run_fwd(p, len, k * p->S, s);
    if (st != MC_OK) return st;
  }
  // final state back to the caller
  auto back = [&](void* dst, const mc_grad_plan::R& r, size_t n) -> cudaError_t {
    if (!dst || n == 0) return cudaSuccess;
    return cudaMemcpyAsync(dst, w + r.off, n, cudaMemcpyDeviceToDevice, s);
  };
  GC(back(state->position, p->r_wpos, (size_t)D.N * 8));
  GC(back(state->velocity, p->r_wvel, (size_t)D.N * 8));
  GC(back(state->theta, p->r_wth, (size_t)D.E * 4));
  GC(back(state->bending_rest_angles, p->r_wra, (size_t)D.B * 4));
  GC(back(state->steric, p->r_wst, HW * 4));
  GC(back(state->fluid_velocity, p->r_wfu, 2 * LHW * 4));
  GC(back(state->f_grid, p->r_wf, 9 * LHW * 4));
  GC(cudaGetLastError());
  p->have_forward = true;
  return MC_OK;
}

mc_status mc_grad_backward(mc_grad_plan* p, const mc_state_cot* final_cot, mc_state_cot* initial_cot,
                           mc_param_grads* grads, void* stream) {
  mc::set_last_error("");
  if (!p || !final_cot || !initial_cot) return gfail(MC_ERR_INVALID, "null argument");
  if (!p->bound) return gfail(MC_ERR_NOT_BOUND, "mc_grad_plan_bind() was not called");
  if (!p->have_forward) return gfail(MC_ERR_INVALID, "mc_grad_forward() has not run on this plan");
  cudaStream_t s = (cudaStream_t)stream;
  const mc_dims& D = p->dims;
  const size_t HW = (size_t)D.H * D.W;
  const size_t LHW = (size_t)p->ad.lHW;  // fluid lattice cells
  unsigned char* w = p->ws;
  AD& d = p->ad;
  auto seed = [&](const mc_grad_plan::R& r, const float* src, size_t n) -> cudaError_t {
    if (n == 0) return cudaSuccess;
    if (!src) return cudaMemsetAsync(w + r.off, 0, n, s);
    return cudaMemcpyAsync(w + r.off, src, n, cudaMemcpyDeviceToDevice, s);
  };
  GC(seed(p->r_lpos, final_cot->position, (size_t)D.N * 8));
  GC(seed(p->r_lvel, final_cot->velocity, (size_t)D.N * 8));
  GC(seed(p->r_lth, final_cot->theta, (size_t)D.E * 4));
  GC(seed(p->r_lf0, final_cot->f_grid, 9 * LHW * 4));
  for (const mc_grad_plan::R* r : {&p->r_dc, &p->r_da, &p->r_dp, &p->r_do, &p->r_dr, &p->r_dl, &p->r_dk})
    GC(cudaMemsetAsync(w + r->off, 0, r->bytes, s));
  if (d.steric && !p->filter_ready) {
    // the forward plan's descriptor exists once mc_grad_forward has run a rollout call
    GC(mc::filter_prepare(p->fwd, w + p->r_fdesc.off, d.lV, d.ctmp, d.ldep, s));
    p->filter_ready = true;
  }
  ++p->backwards;
  int lfcur = 0;
  // Replay of segment k - 1 beside the reverse of segment k: a replayed step keeps one SM busy for
  // most of its time and a reverse step a few, and they share nothing but the two copies of the
  // segment's inputs.  48 steps at 256^2 21.5 -> 16.9 ms, 12 at 640^2 10.2 -> 9.5.
  cudaStream_t rs = p->overlap ? p->replay_stream : s;
  auto after = [&](cudaEvent_t ev, cudaStream_t from, cudaStream_t to) {
    cudaError_t e = cudaEventRecord(ev, from);
    return e == cudaSuccess ? cudaStreamWaitEvent(to, ev, 0) : e;
  };
  if (p->overlap) GC(after(p->ev_begin, s, rs));
  // whatever happens, the caller's stream waits for the replay's
  struct Join {
    mc_grad_plan* p;
    cudaStream_t from, to;
    ~Join() {
      if (from != to && cudaEventRecord(p->ev_begin, from) == cudaSuccess) cudaStreamWaitEvent(to, p->ev_begin, 0);
    }
  } join{p, rs, s};
  mc_status st = p->nseg > 0 ? replay_segment(p, p->nseg - 1, rs) : MC_OK;
  if (st != MC_OK) return st;
  for (int k = p->nseg - 1; k >= 0; --k) {
    const int t0 = k * p->S;
    const int len = std::min(p->S, p->T - t0);
    if (p->overlap) {
      GC(after(p->ev_replayed[k & 1], rs, s));
      if (k > 0) {
        // segment k - 1 goes where segment k + 1 was
        if (k + 1 < p->nseg) GC(cudaStreamWaitEvent(rs, p->ev_reversed[(k + 1) & 1], 0));
        st = replay_segment(p, k - 1, rs);
        if (st != MC_OK) return st;
      }
    } else if (k < p->nseg - 1) {
      st = replay_segment(p, k, s);
      if (st != MC_OK) return st;
    }
    // per-step inputs of the segment (the cotangent of f alternates between two buffers)
    p->sargs.assign(len, StepArgs{});
    for (int j = len - 1; j >= 0; --j) {
      const int at_j = segment_slot(p, k, j);
      Slot sj = slot(p, p->r_seg, at_j);
      StepArgs& a = p->sargs[j];
      a.t = t0 + j;
      a.pos = sj.pos;
      a.vel = sj.vel;
      a.th = sj.th;
      a.f = sj.f;
      a.V = reinterpret_cast<const float*>(w + p->r_segV.off + (size_t)at_j * al(HW * 4));
      a.lf_in = at<float>(w, lfcur ? p->r_lf1 : p->r_lf0);
      a.lf_out = at<float>(w, lfcur ? p->r_lf0 : p->r_lf1);
      if (d.fluid) lfcur ^= 1;
    }
    const int jlast = len - 1, jp[2] = {jlast, jlast - 1};
    {
      // staged: the host arrays may change once the call returns, and the host does not
      // wait here for the stream to reach these copies
      const mc::Upload u[2] = {{w + p->r_sargs.off, p->sargs.data(), len * sizeof(StepArgs)},
                               {w + p->r_jp.off, jp, sizeof(jp)}};
      GC(mc::stage_uploads(u, 2, s));
    }
    if (p->rev_graph_act != d.has_act) drop_rev_graphs(p);
    p->rev_graph_act = d.has_act;
    auto run = [&](int which) -> mc_status {
      if (!reverse_graphs(p)) {
        enqueue_reverse(p, which, s);
        return MC_OK;
      }
      cudaGraphExec_t g;
      mc_status gs = rev_graph(p, which, &g);
      if (gs == MC_OK) GC(cudaGraphLaunch(g, s));
      return gs;
    };
    if (p->tape_bytes) {
      st = run(jlast & 1 ? kTapeOdd : kTapeEven);
      for (int j = jlast; j > 0 && st == MC_OK; --j) st = run(j & 1 ? kBothOdd : kBothEven);
      if (st == MC_OK) st = run(kReverseEven);
    } else {
      for (int j = jlast; j >= 0 && st == MC_OK; --j) st = run(kWhole);
    }
    if (st != MC_OK) return st;
    GC(cudaGetLastError());
    if (p->overlap) GC(cudaEventRecord(p->ev_reversed[k & 1], s));
  }
  auto out = [&](float* dst, const mc_grad_plan::R& r, size_t n) -> cudaError_t {
    if (!dst || n == 0) return cudaSuccess;
    return cudaMemcpyAsync(dst, w + r.off, n, cudaMemcpyDeviceToDevice, s);
  };
  GC(out(initial_cot->position, p->r_lpos, (size_t)D.N * 8));
  GC(out(initial_cot->velocity, p->r_lvel, (size_t)D.N * 8));
  GC(out(initial_cot->theta, p->r_lth, (size_t)D.E * 4));
  GC(out(initial_cot->f_grid, lfcur ? p->r_lf1 : p->r_lf0, 9 * LHW * 4));
  if (grads) {
    GC(out(grads->act_c, p->r_dc, (size_t)D.B * 4));
    GC(out(grads->act_amp, p->r_da, (size_t)D.B * 4));
    GC(out(grads->act_phase, p->r_dp, (size_t)D.B * 4));
    GC(out(grads->act_omega, p->r_do, (size_t)D.B * 4));
    GC(out(grads->rest_angles, p->r_dr, (size_t)D.B * 4));
    GC(out(grads->rest_lengths, p->r_dl, (size_t)D.E * 4));
    GC(out(grads->bending_stiffness, p->r_dk, (size_t)D.B * 4));
  }
  GC(cudaGetLastError());
  return MC_OK;
}

}  // extern "C"
