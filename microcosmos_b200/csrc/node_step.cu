// The node side of a whole step in one launch, one CTA per rollout, for plans whose rollouts are
// small enough to keep their IB stencils in shared memory ("compact" plans, runtime.cu):
//
//   steric displacement of the prediction   (forces.py:41-81, simulate.py:46-65)
//   rod iterations                          (rod.cuh)
//   velocity, IB stencils, touched cells    (simulate.py:83-84, fluid.py:40-79, 268-290)
//   multi-direct forcing, body force        (fluid.py:292-339)
//   node reaction, wrap, recording          (fluid.py:359-382, simulate.py:97-98)
//   the next step's cloud-in-cell deposit   (forces.py:84-115)
//
// What bounds these rollouts is the number of dependent launches: as separate kernels this is a
// chain of 19, each a few microseconds of launch, descriptor and index loads for less than a
// microsecond of work.  In one CTA the phases are separated by barriers, and everything that one
// phase hands to the next (positions, stencil weights, the touched cells' velocities, the
// corrections) stays in shared memory.  Every sum runs over the same operands in the same order as
// in the separate kernels, so the results are the same bits.
#include "rod.cuh"

#include "node_step.cuh"

namespace mc {

namespace {

using u16 = unsigned short;

extern __shared__ __align__(16) unsigned char node_smem[];

// The CTA's shared memory, laid out by NodeStepShape: arrays per node, per IB point, per
// contribution, per touched cell, and a region whose uses follow one another (rod tables; hash of
// the cells; unsorted runs; the touched cells' velocities).  Addresses are formed where they are
// used, from the kernel's parameters.
struct Smem {
  const NodeStepShape& s;
  template <typename T>
  __device__ __forceinline__ static T* at(int off) {
    return reinterpret_cast<T*>(node_smem + off);
  }
  __device__ __forceinline__ float* pos() const { return at<float>(s.pos); }        // N x 2
  __device__ __forceinline__ float* vel() const { return at<float>(s.vel); }        // N x 2
  __device__ __forceinline__ float2* nvl() const { return at<float2>(s.nvl); }      // NI: lattice velocity of the point
  __device__ __forceinline__ float2* delta() const { return at<float2>(s.delta); }  // NI: its current correction
  // contributions: weights entry-major (stencil entry e of point p at e * NI + p), touched cell
  __device__ __forceinline__ float* w() const { return at<float>(s.w); }
  __device__ __forceinline__ u16* slot() const { return at<u16>(s.slot); }
  // runs: weights (before the sort: the contributions' cells) and points
  __device__ __forceinline__ float* rw() const { return at<float>(s.rw); }
  __device__ __forceinline__ int* cell() const { return at<int>(s.rw); }
  __device__ __forceinline__ u16* rn() const { return at<u16>(s.rn); }
  // touched cells: cell, then 1 / max(coverage, 1); start << 16 | length of the run
  __device__ __forceinline__ int* hcell() const { return at<int>(s.hcell); }
  __device__ __forceinline__ float* inv() const { return at<float>(s.hcell); }
  __device__ __forceinline__ unsigned* hrun() const { return at<unsigned>(s.hrun); }
  // one region: rod tables; hash (cell or -1; first contribution, then touched cell); runs in
  // arrival order; the touched cells' corrected velocity, then body force
  __device__ __forceinline__ float2* tab() const { return at<float2>(s.shared); }
  __device__ __forceinline__ int* key() const { return at<int>(s.shared); }
  __device__ __forceinline__ int* owner() const { return at<int>(s.shared + 4 * s.hash); }
  __device__ __forceinline__ int* count() const { return at<int>(s.hcell); }  // hash: contributions (before hcell, hrun)
  __device__ __forceinline__ u16* raw() const { return at<u16>(s.shared); }
  __device__ __forceinline__ float2* uc() const { return at<float2>(s.shared); }
};

// index wrapped into [0, m): one addition for the neighbouring period, the general modulo beyond
__device__ __forceinline__ int wrap_index(int i, int m) {
  int r = i < 0 ? i + m : (i >= m ? i - m : i);
  return (unsigned)r < (unsigned)m ? r : imod_floor(i, m);
}

// Inertial prediction of a node from its position and velocity (simulate.py:46-50), and wrapped.
struct Predicted {
  float qx, qy, wx, wy;
};
__device__ __forceinline__ Predicted predict(const RDesc& d, float px, float py, float vx, float vy) {
  Predicted p;
  p.qx = px + (vx * d.damping) * d.dt;
  p.qy = py + (vy * d.damping) * d.dt;
  p.wx = fmod_floor(p.qx, (float)d.W);
  p.wy = fmod_floor(p.qy, (float)d.H);
  return p;
}

// map_coordinates(V, [yy, xx], order=1, mode="wrap") (forces.py:30-34)
__device__ __forceinline__ float sample(const float* __restrict__ V, int H, int W, float yy, float xx) {
  const float ly = floorf(yy), lx = floorf(xx);
  const float ty = yy - ly, tx = xx - lx;
  const float wy0 = 1.0f - ty, wx0 = 1.0f - tx;
  const int iy0 = wrap_index((int)ly, H), iy1 = wrap_index((int)ly + 1, H);
  const int ix0 = wrap_index((int)lx, W), ix1 = wrap_index((int)lx + 1, W);
  const float a = V[(size_t)iy0 * W + ix0], b = V[(size_t)iy0 * W + ix1];
  const float c = V[(size_t)iy1 * W + ix0], e = V[(size_t)iy1 * W + ix1];
  float acc = (wy0 * wx0) * a;
  acc = acc + (wy0 * tx) * b;
  acc = acc + (ty * wx0) * c;
  acc = acc + (ty * tx) * e;
  return acc;
}

// The four cells and weights of a node's cloud-in-cell deposit (forces.py:98-115), corner c:
// (y0, x0), (y0, x1), (y1, x0), (y1, x1).
__device__ __forceinline__ int cic_cell(const RDesc& d, const Predicted& p, int c, float& w) {
  const float fx = floorf(p.wx), fy = floorf(p.wy);
  const int x0 = wrap_index((int)fx, d.W), y0 = wrap_index((int)fy, d.H);
  const int x1 = x0 + 1 == d.W ? 0 : x0 + 1, y1 = y0 + 1 == d.H ? 0 : y0 + 1;
  const float dx = p.wx - fx, dy = p.wy - fy;
  const float ax = (c & 1) ? dx : 1.0f - dx, ay = (c & 2) ? dy : 1.0f - dy;
  w = (ax * ay) * d.st_scatter;
  return ((c & 2) ? y1 : y0) * d.W + ((c & 1) ? x1 : x0);
}

// Sum of `v` over the threads before this one, and over all of them.
__device__ __forceinline__ int scan_threads(int v, int* warp_sum, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  const int ws = lane < warps ? warp_sum[lane] : 0;
  total = __reduce_add_sync(0xffffffffu, ws);
  return __reduce_add_sync(0xffffffffu, lane < warp ? ws : 0) + incl - v;
}

// Groups n contributions by cell.  In: their cells and weights.  Out: each contribution's touched
// cell (slot), and every touched cell's run of (point, weight) in the order of the reference's
// scatter, its start and length, and its cell; returns the number of touched cells.  They are
// numbered by their first contribution in scatter order, so that neighbours on a rod are
// neighbours in memory: the accesses to the populations that follow then share their sectors.
// place(k): where the k-th contribution of the scatter order is kept; point(k): its point.
template <typename Place, typename Point>
__device__ __forceinline__ int group_by_cell(const Smem& m, int n, int* warp_sum, Place place, Point point) {
  const int tid = threadIdx.x, T = blockDim.x, hash = m.s.hash;
  int* const key = m.key();
  int* const owner = m.owner();
  int* const count = m.count();
  const int* const cell = m.cell();
  u16* const slot = m.slot();
  u16* const rn = m.rn();
  unsigned* const hrun = m.hrun();
  for (int i = tid; i < hash / 4; i += T) {
    reinterpret_cast<int4*>(key)[i] = make_int4(-1, -1, -1, -1);
    reinterpret_cast<int4*>(owner)[i] = make_int4(n, n, n, n);
    reinterpret_cast<int4*>(count)[i] = make_int4(0, 0, 0, 0);
  }
  __syncthreads();
  for (int k = tid; k < n; k += T) {
    const int at = place(k), c = cell[at];
    unsigned e = __umulhi((unsigned)c * 2654435761u, (unsigned)hash);
    for (;;) {  // ends: there are more entries than contributions
      const int old = atomicCAS(key + e, -1, c);
      if (old == -1 || old == c) break;
      e = e + 1 == (unsigned)hash ? 0u : e + 1;
    }
    atomicMin(owner + e, k);
    atomicAdd(count + e, 1);
    slot[at] = (u16)e;
  }
  __syncthreads();
  // number the cells by their owners in scatter order, and place their runs: a stretch of the
  // contributions per thread (low half: cells, high half: length of their runs)
  const int per = (n + T - 1) / T, a = min(tid * per, n), b = min(a + per, n);
  int sum = 0, all;
  for (int k = a; k < b; ++k) {
    const int e = slot[place(k)], len = owner[e] == k ? count[e] : 0;
    rn[k] = (u16)len;
    sum += len > 0 ? 1 + (len << 16) : 0;
  }
  sum = scan_threads(sum, warp_sum, all);
  const int heads = all & 0xffff;
  for (int k = a; k < b; ++k) {
    const int len = rn[k];
    if (len > 0) {
      const int at = place(k), h = sum & 0xffff;
      owner[slot[at]] = h;
      m.hcell()[h] = cell[at];
      hrun[h] = (unsigned)sum & 0xffff0000u;
      sum += 1 + (len << 16);
    }
  }
  __syncthreads();
  u16* const raw = m.raw();
  for (int k = tid; k < n; k += T) {
    const int at = place(k), h = owner[slot[at]];
    slot[at] = (u16)h;
    const unsigned r = atomicAdd(hrun + h, 1u);
    raw[(r >> 16) + (r & 0xffffu)] = (u16)k;
  }
  __syncthreads();
  const float* const w = m.w();
  float* const rw = m.rw();
  for (int k = tid; k < n; k += T) {
    const int at = place(k);
    const unsigned r = hrun[slot[at]];
    const int start = (int)(r >> 16), len = (int)(r & 0xffffu);
    int rank = 0;
    for (int q = 0; q < len; ++q) rank += raw[start + q] < k ? 1 : 0;
    rn[start + rank] = (u16)point(k);
    rw[start + rank] = w[at];
  }
  __syncthreads();
  return heads;
}

// One point's stencil: its touched cells (two to a register) and weights.
template <int K2>
struct Stencil {
  unsigned slot[(K2 + 1) / 2];
  float w[K2];
  __device__ __forceinline__ void load(const Smem& m, int NI, int p) {
#pragma unroll
    for (int s = 0; s < K2; ++s) {
      const unsigned h = m.slot()[s * NI + p];
      if (s & 1)
        slot[s / 2] |= h << 16;
      else
        slot[s / 2] = h;
      w[s] = m.w()[s * NI + p];
    }
  }
  // sum of uc(touched cell) * weight, in stencil order
  __device__ __forceinline__ float2 sum(const float2* uc) const {
    float2 v[K2];
#pragma unroll
    for (int s = 0; s < K2; ++s) v[s] = uc[(s & 1) ? slot[s / 2] >> 16 : slot[s / 2] & 0xffffu];
    float x = 0.0f, y = 0.0f;
#pragma unroll
    for (int s = 0; s < K2; ++s) {
      x = x + v[s].x * w[s];
      y = y + v[s].y * w[s];
    }
    return make_float2(x, y);
  }
};

// The multi-direct forcing rounds (fluid.py:292-310), the body force of each touched cell
// (fluid.py:327-339) and each point's share of it (fluid.py:364-370, in the place of delta).  A
// thread keeps its first point's stencil in registers for all rounds.
template <int K2>
__device__ __forceinline__ void forcing(const RDesc& d, const Smem& m, int NI, int heads) {
  const int tid = threadIdx.x, T = blockDim.x;
  const float vmax = d.vmax, q4 = d.vmax_q4, relax = d.relax;
  const int iters = d.ib_iters, clamp_force = d.force_clamp;
  const float4* __restrict__ s_mac = d.s_mac;
  float2* __restrict__ s_f = d.s_f;
  const float* const inv = m.inv();
  float2* const uc = m.uc();
  float2* const delta = m.delta();
  const float2* const nvl = m.nvl();
  const unsigned* const hrun = m.hrun();
  const u16* const rn = m.rn();
  const float* const rw = m.rw();
  Stencil<K2> st;
  if (tid < NI) st.load(m, NI, tid);
  for (int it = 0; it < iters; ++it) {
    for (int p = tid; p < NI; p += T) {
      if (p != tid) st.load(m, NI, p);
      const float2 u = st.sum(uc), v = nvl[p];
      const float sx = (v.x - u.x) * relax, sy = (v.y - u.y) * relax;
      const float cf = clamp_factor_fast(sx, sy, vmax, q4);
      delta[p] = make_float2(sx * cf, sy * cf);
    }
    if (tid + T < NI) st.load(m, NI, tid);
    __syncthreads();
    for (int h = tid; h < heads; h += T) {
      const unsigned run = hrun[h];
      const int start = (int)(run >> 16), len = (int)(run & 0xffffu);
      float dx = 0.0f, dy = 0.0f;
      // the loads of 4 entries are in flight together, the sums keep the run order; entries
      // beyond the run are not loaded (the shared-memory accesses of all warps share one pipe)
      for (int j = 0; j < len; j += 4) {
        float2 e[4];
        float w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (j + q < len) {
            e[q] = delta[rn[start + j + q]];
            w[q] = rw[start + j + q];
          }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (j + q < len) {
            dx = dx + e[q].x * w[q];
            dy = dy + e[q].y * w[q];
          }
      }
      const float2 u = uc[h];
      const float iv = inv[h];
      uc[h] = make_float2(u.x + dx * iv, u.y + dy * iv);
    }
    __syncthreads();
  }
  for (int h = tid; h < heads; h += T) {
    float2 u = uc[h];
    const float4 mac = s_mac[h];
    const float c2 = clamp_factor_fast(u.x, u.y, vmax, q4);
    u.x = u.x * c2;
    u.y = u.y * c2;
    float Fx = (u.x - mac.y) * mac.x, Fy = (u.y - mac.z) * mac.x;
    if (clamp_force) {
      const float c3 = clamp_factor(Fx, Fy, vmax);
      Fx = Fx * c3;
      Fy = Fy * c3;
    }
    s_f[h] = make_float2(Fx, Fy);
    uc[h] = make_float2(Fx, Fy);
  }
  __syncthreads();
  for (int p = tid; p < NI; p += T) {
    if (p != tid) st.load(m, NI, p);
    delta[p] = st.sum(uc);
  }
}

// The coupling of the IB points, whose stencils are ready, with the fluid: touched cells with their
// coverage and macroscopic state (fluid.py:268-290), then the forcing.
template <int K>
__device__ __forceinline__ void couple(const RDesc& d, const Smem& m, int* warp_sum, int parity) {
  constexpr int K2 = K * K;
  const int tid = threadIdx.x, T = blockDim.x, NI = d.NI;
  const int heads =
      group_by_cell(m, d.M, warp_sum, [=](int k) { return (k % K2) * NI + k / K2; }, [](int k) { return k / K2; });
  const float* __restrict__ hp = d.h[parity];
  const int lW = d.lW, lH = d.lH;
  const size_t HW = (size_t)lH * lW;
  const float vmax = d.vmax, q4 = d.vmax_q4;
  int* __restrict__ h_cell = d.h_cell;
  float4* __restrict__ s_mac = d.s_mac;
  if (tid == 0) d.ib_ctl[5] = heads;  // for k_collide_heads
  for (int h = tid; h < heads; h += T) {
    const int cell = m.hcell()[h];
    const int y = cell / lW, x = cell - y * lW;
    const int xm = x == 0 ? lW - 1 : x - 1, xp = x == lW - 1 ? 0 : x + 1;
    const float* r0 = hp + (size_t)y * lW;  // populations are pulled from the cell opposite to their direction
    const float* rm = hp + (size_t)(y == 0 ? lH - 1 : y - 1) * lW;
    const float* rp = hp + (size_t)(y == lH - 1 ? 0 : y + 1) * lW;
    float f[9];
    f[0] = r0[x];
    f[1] = r0[HW + xm];
    f[2] = rm[2 * HW + x];
    f[3] = r0[3 * HW + xp];
    f[4] = rp[4 * HW + x];
    f[5] = rm[5 * HW + xm];
    f[6] = rm[6 * HW + xp];
    f[7] = rp[7 * HW + xp];
    f[8] = rp[8 * HW + xm];
    const unsigned run = m.hrun()[h];
    const int start = (int)(run >> 16), len = (int)(run & 0xffffu);
    float cov = m.rw()[start];
    for (int q = 1; q < len; ++q) cov = cov + m.rw()[start + q];
    float rho, vx, vy;
    macroscopic(f, vmax, q4, rho, vx, vy);
    h_cell[h] = cell;
    const float inv = 1.0f / max_prop(cov, 1.0f);
    s_mac[h] = make_float4(rho, vx, vy, 0.0f);
    m.inv()[h] = inv;
    m.uc()[h] = make_float2(vx, vy);
  }
  __syncthreads();
  forcing<K2>(d, m, NI, heads);
}

// IB point p of a node at (x, y) in lattice units (fluid.py:236-263, as ib_point in pbd.cu).
__device__ __forceinline__ float2 lattice_point(const RDesc& d, const float* pos, int p, int node, float x, float y) {
  const float gx = x * d.scale_x, gy = y * d.scale_y;
  if (!(d.syn_w > 0.0f)) return make_float2(gx, gy);
  float tx = 0.0f, ty = 0.0f;
  for (int j = d.ne_off[node]; j < d.ne_off[node + 1]; ++j) {
    const int e = d.ne_idx[j] >> 1;
    const int s = d.pairs[2 * e], g = d.pairs[2 * e + 1];
    const float2 ev = min_image(pos[2 * g], pos[2 * g + 1], pos[2 * s], pos[2 * s + 1], (float)d.W, (float)d.H);
    tx = tx + ev.x;
    ty = ty + ev.y;
  }
  const float nrm = sqrtf((tx * tx + ty * ty) + MC_EPSIL);
  const float ux = tx / nrm, uy = ty / nrm;
  const float ox = (d.syn_w * (-uy)) * d.syn_ms, oy = (d.syn_w * ux) * d.syn_ms;
  return p < d.N ? make_float2(gx + ox, gy + oy) : make_float2(gx - ox, gy - oy);
}

}  // namespace

// main: the step itself; next: the following step's deposit (a rollout's first launch has next
// alone, its last main alone).  tdev[r]: rollout r's step counter, advanced here.
__global__ void __launch_bounds__(kNodeStepMaxThreads, 1)
    k_node_step(const RDesc* __restrict__ D, int* __restrict__ tdev, const __grid_constant__ NodeStepShape shape, int parity, int main,
                int next) {
  __shared__ __align__(16) unsigned char desc_bytes[sizeof(RDesc)];
  __shared__ int warp_sum[kNodeStepMaxThreads / 32];
  const int r = blockIdx.x;
  const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5;
  // the descriptor, once: its fields are used in every phase
  {
    static_assert(sizeof(RDesc) % 4 == 0, "copied by words");
    const unsigned* src = reinterpret_cast<const unsigned*>(D + r);
    unsigned* dst = reinterpret_cast<unsigned*>(desc_bytes);
    for (int i = tid; i < (int)(sizeof(RDesc) / 4); i += T) dst[i] = src[i];
  }
  const int t = tdev[r];
  __syncthreads();
  const RDesc& d = *reinterpret_cast<const RDesc*>(desc_bytes);
  const Smem m{shape};
  const int N = d.N, NI = d.NI;
  const float Wf = (float)d.W, Hf = (float)d.H;

  if (main) {
    // ---- prediction; its wrapped form stays in the place of the velocities for the neighbours
    for (int i = tid; i < N; i += T) {
      const Predicted p = predict(d, d.pos[2 * i], d.pos[2 * i + 1], d.vel[2 * i], d.vel[2 * i + 1]);
      m.pos()[2 * i] = p.qx;
      m.pos()[2 * i + 1] = p.qy;
      m.vel()[2 * i] = p.wx;
      m.vel()[2 * i + 1] = p.wy;
    }
    __syncthreads();
    if (d.enable_steric) {
      // ---- steric displacement: 4 lanes per node, one finite-difference sample and a quarter of
      // the neighbours each
      const float* __restrict__ V = d.steric;
      float* __restrict__ dep = d.dep;
      const int H = d.H, W = d.W, nsk = d.st_skip;
      const float two_s2 = d.st_2s2, norm = d.st_norm, coef = d.st_coef, strength = d.st_strength, dt = d.dt;
      const unsigned full = 0xffffffffu;
      for (int i0 = 0; i0 < N; i0 += T / 4) {
        const int i = i0 + (tid >> 2), q = tid & 3;
        const int node = min(i, N - 1);
        Predicted p;
        p.qx = m.pos()[2 * node];
        p.qy = m.pos()[2 * node + 1];
        p.wx = m.vel()[2 * node];
        p.wy = m.vel()[2 * node + 1];
        float wgt;
        const int cell = cic_cell(d, p, q, wgt);
        const float half = (q & 1) ? -0.5f : 0.5f;
        const float v = sample(V, H, W, q < 2 ? p.wy : p.wy + half, q < 2 ? p.wx + half : p.wx);
        if (i < N) dep[cell] = 0.0f;  // the deposit grid stays zero between steps
        const float xp = __shfl_sync(full, v, 0, 4), xm = __shfl_sync(full, v, 1, 4);
        const float yp = __shfl_sync(full, v, 2, 4), ym = __shfl_sync(full, v, 3, 4);
        float fx = -((xp - xm) / 1.0f), fy = -((yp - ym) / 1.0f);
        if (nsk > 0) {
          float ax = 0.0f, ay = 0.0f;
          for (int o = -nsk; o <= nsk; o += 4) {
            const int j = node + o + q;
            const bool there = j >= 0 && j < N && o + q <= nsk;
            float tx = 0.0f, ty = 0.0f;
            if (there && j != node) {  // a node's own term is zero
              const float2 rr = min_image(p.wx, p.wy, m.vel()[2 * j], m.vel()[2 * j + 1], Wf, Hf);
              const float d2 = rr.x * rr.x + rr.y * rr.y;
              const float kv = expf(-d2 / two_s2) / norm;
              tx = kv * rr.x;
              ty = kv * rr.y;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              ax = ax + __shfl_sync(full, tx, e, 4);
              ay = ay + __shfl_sync(full, ty, e, 4);
            }
          }
          fx = fx - coef * ax;
          fy = fy - coef * ay;
        }
        if (q == 0 && i < N) {
          m.pos()[2 * i] = p.qx + (fx * strength) * dt;
          m.pos()[2 * i + 1] = p.qy + (fy * strength) * dt;
        }
      }
      __syncthreads();
    }
    // ---- rods: teams of the same number of warps, one rod at a time each
    {
      const int tw = shape.rod_warps, team = warp / tw;
      const Team tm = {warp - team * tw, tw, 1 + shape.bars * team};
      if (team < shape.teams)
        for (int c = team; c < d.nchain; c += shape.teams) {
          // all warps of the team, those that the rod before did not use too
          if (c != team && d.solver == 1) tm.sync();
          chain_rod<false>(d, d.chain_info[c], t, tm, m.pos(), m.tab() + (size_t)team * chain_smem(shape.longest),
                           shape.longest);
        }
    }
    __syncthreads();
    // ---- velocity, IB points and their stencils: 4 lanes per IB point, lane a column a of the
    // kernel; the weights' sum is taken in entry order a * K + b
    const int K = d.K;
    {
      const int hk = (K - 1) / 2, a = tid & 3;
      const float hw = (float)K / 2.0f, dt = d.dt, scx = d.scale_x, scy = d.scale_y;
      const int lW = d.lW, lH = d.lH, fluid = d.enable_fluid;
      const float* __restrict__ pos = d.pos;
      const unsigned full = 0xffffffffu;
      int* const cells = m.cell();
      const int points = max(N, NI);
      for (int p0 = 0; p0 < points; p0 += T / 4) {
        const int p = min(p0 + (tid >> 2), points - 1);
        const bool on = p0 + (tid >> 2) < points;
        const int node = p < N ? p : p - N;
        const float x = m.pos()[2 * node], y = m.pos()[2 * node + 1];
        const float vx = (x - pos[2 * node]) / dt, vy = (y - pos[2 * node + 1]) / dt;
        if (on && a == 0) {
          if (p < N) {
            m.vel()[2 * node] = vx;
            m.vel()[2 * node + 1] = vy;
          }
          m.nvl()[p] = make_float2((vx * scx) * dt, (vy * scy) * dt);
        }
        if (!fluid) continue;
        const float2 g = lattice_point(d, m.pos(), p, node, x, y);
        const float bx = (floorf(g.x) - (float)hk) + (float)a, by = (floorf(g.y) - (float)hk) + (float)a;
        const float rx = fabsf(bx - g.x) / hw, ry = fabsf(by - g.y) / hw;
        const float wxa = rx <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * rx) / 2.0f)) : 0.0f;
        const float wya = ry <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * ry) / 2.0f)) : 0.0f;
        const int cx = wrap_index((int)bx, lW), cya = wrap_index((int)by, lH) * lW;
        float w[4];
        int row[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          w[b] = wxa * __shfl_sync(full, wya, b, 4);
          row[b] = __shfl_sync(full, cya, b, 4);
        }
        float sum = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const float we = __shfl_sync(full, w[b], e, 4);
            if (e < K && b < K) sum = sum + we;
          }
        if (on && a < K) {
          const float den = sum + MC_EPSIL;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (b < K) {
              const int at = (a * K + b) * NI + p;
              m.w()[at] = w[b] / den;
              cells[at] = row[b] + cx;
            }
        }
      }
    }
    __syncthreads();
    if (d.enable_fluid) {
      if (K == 4)
        couple<4>(d, m, warp_sum, parity);
      else if (K == 3)
        couple<3>(d, m, warp_sum, parity);
      else if (K == 2)
        couple<2>(d, m, warp_sum, parity);
      else
        couple<1>(d, m, warp_sum, parity);
      __syncthreads();
    }
    // ---- node reaction (fluid.py:364-382), wrap (simulate.py:97-98), flags, recording
    for (int i = tid; i < N; i += T) {
      float vx = m.vel()[2 * i], vy = m.vel()[2 * i + 1];
      if (d.enable_fluid) {
        float2 f = m.delta()[i];
        if (NI > N) {
          const float2 g = m.delta()[i + N];
          f = make_float2(0.5f * (f.x + g.x), 0.5f * (f.y + g.y));
        }
        vx = vx - (f.x / d.node_mass) / d.sdt_x;
        vy = vy - (f.y / d.node_mass) / d.sdt_y;
      }
      const float px = fmod_floor(m.pos()[2 * i], Wf), py = fmod_floor(m.pos()[2 * i + 1], Hf);
      d.vel[2 * i] = vx;
      d.vel[2 * i + 1] = vy;
      d.pos[2 * i] = px;
      d.pos[2 * i + 1] = py;
      if (!(isfinite(px) && isfinite(py) && isfinite(vx) && isfinite(vy))) atomicOr(d.flags, 1u);
      if (d.rec_every > 0 && (t + 1) % d.rec_every == 0) {
        const size_t e = (size_t)((t + 1) / d.rec_every - 1) * N * 2;
        if (d.rec_pos) {
          d.rec_pos[e + 2 * i] = px;
          d.rec_pos[e + 2 * i + 1] = py;
        }
        if (d.rec_vel) {
          d.rec_vel[e + 2 * i] = vx;
          d.rec_vel[e + 2 * i + 1] = vy;
        }
      }
    }
    if (tid == 0) tdev[r] = t + 1;
    __syncthreads();
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the filter's CTAs may come and wait

  if (next && d.enable_steric) {
    int* const cell = m.cell();
    for (int c = tid; c < 4 * N; c += T) {
      const int corner = c / N, i = c - corner * N;
      const Predicted p = predict(d, d.pos[2 * i], d.pos[2 * i + 1], d.vel[2 * i], d.vel[2 * i + 1]);
      float w;
      cell[c] = cic_cell(d, p, corner, w);
      m.w()[c] = w;
    }
    __syncthreads();
    const int heads =
        group_by_cell(m, 4 * N, warp_sum, [](int k) { return k; }, [](int k) { return k; });
    for (int h = tid; h < heads; h += T) {
      const unsigned run = m.hrun()[h];
      const int start = (int)(run >> 16), len = (int)(run & 0xffffu);
      float acc = m.rw()[start];
      for (int q = 1; q < len; ++q) acc = acc + m.rw()[start + q];
      d.dep[m.hcell()[h]] = acc;
    }
  }
}

void launch_node_step(const RDesc* d, int n, int* tdev, const NodeStepShape& shape, int parity, int main, int next,
                      cudaStream_t s) {
  k_node_step<<<n, shape.threads, shape.bytes, s>>>(d, tdev, shape, parity, main, next);
}
cudaError_t node_step_set_smem(size_t bytes) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_node_step);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_node_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes - a.sharedSizeBytes));
}

}  // namespace mc
