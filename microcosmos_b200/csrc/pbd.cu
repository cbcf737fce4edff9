// Node-side kernels of one step (src/microcosmos/simulate.py:37-84):
//   k_predict: damping, inertial prediction, steric cloud-in-cell contributions;
//   k_steric:  per node, the steric force added to the prediction (forces.py:41-81);
//   k_chain:   one CTA per chain rod (the topology make_edges(.., "line", F) builds),
//              one node per lane, neighbours exchanged with shuffles (rod.cuh);
//   k_node:    one CTA per rod of any other topology (trees, loops), state in shared
//              memory, scatter-adds as gather lists in the reference's order.
//   k_stencil: per node, the velocity from positions and the IB stencil (fluid.py:40-87).
// Both rod kernels evaluate the curvature actuation and run cycles_per_step Jacobi
// iterations of pbd_rod_constraint (solver/pbd.py:14-91).
#include "rod.cuh"

namespace mc {

__device__ __forceinline__ int bin_tile(const RDesc& d, int cy, int cx) {
  return (cy / kBinTile) * d.ntile_x + cx / kBinTile;
}

__global__ void __launch_bounds__(256) k_predict(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                 int* tdev) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int node = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  if (tdev && blockIdx.x == 0 && threadIdx.x == 0) *tdev += 1;  // the step before ends here
  if (node == 0) {
    // the previous step's IB work is complete: reset this step's IB controls
    d.ib_ctl[0] = 0;
    d.ib_ctl[1] = 0;
    d.ib_ctl[2] = 0;
  }
  if (node >= d.N) return;
  const float px = d.pos[2 * node], py = d.pos[2 * node + 1];
  const float vx = d.vel[2 * node] * d.damping, vy = d.vel[2 * node + 1] * d.damping;
  d.prev[2 * node] = px;
  d.prev[2 * node + 1] = py;
  d.vel[2 * node] = vx;
  d.vel[2 * node + 1] = vy;
  const float qx = px + vx * d.dt, qy = py + vy * d.dt;
  d.pred[2 * node] = qx;
  d.pred[2 * node + 1] = qy;
  if (!d.enable_steric) return;
  // update_steric_potential (forces.py:84-115): CIC weights of the wrapped prediction
  const float W = (float)d.W, H = (float)d.H;
  const float x = fmod_floor(qx, W), y = fmod_floor(qy, H);
  d.predw[2 * node] = x;
  d.predw[2 * node + 1] = y;
  const float fx = floorf(x), fy = floorf(y);
  const int x0 = imod_floor((int)fx, d.W), y0 = imod_floor((int)fy, d.H);
  const int x1 = (x0 + 1) % d.W, y1 = (y0 + 1) % d.H;
  const float dx = x - fx, dy = y - fy;
  const float s = d.st_scatter;
  const float w[4] = {((1.0f - dx) * (1.0f - dy)) * s, (dx * (1.0f - dy)) * s, ((1.0f - dx) * dy) * s, (dx * dy) * s};
  const int cy[4] = {y0, y0, y1, y1};
  const int cx[4] = {x0, x1, x0, x1};
  int tile[4], first[4], cnt[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    tile[c] = bin_tile(d, cy[c], cx[c]);
    first[c] = c;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < c && tile[e] == tile[c] && first[c] == c) first[c] = e;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    cnt[c] = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) cnt[c] += (first[e] == c) ? 1 : 0;
  }
  int base[4], rank[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    base[c] = cnt[c] ? atomicAdd(d.c_tcount + tile[c], cnt[c]) : -1;
    if (base[c] == 0) d.wl_cic[atomicAdd(d.wl_ctl + 1, 1)] = make_int2(d.ridx, tile[c]);
    rank[c] = 0;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int k = c * d.N + node;
    d.c_cell[k] = cy[c] * d.W + cx[c];
    d.c_w[k] = w[c];
    const int g = first[c];
    const int pos = base[g] + rank[g]++;
    if (pos < d.c_cap) {
      d.c_store[(size_t)tile[c] * d.c_cap + pos] = bin_entry(cy[c], cx[c], k);
    } else {
      d.c_ovf[atomicAdd(d.c_ctl, 1)] = k;
    }
  }
}

// One edge force (pbd.py:60-81).
__device__ __forceinline__ float2 edge_force(const RDesc& d, float th, float L0, float xs, float ys, float xt,
                                             float yt) {
  float sn, cs;
  sincosf(th, &sn, &cs);
  const float tx = cs * L0, ty = sn * L0;
  const float2 cur = min_image(xt, yt, xs, ys, (float)d.W, (float)d.H);
  const float L = sqrtf(cur.x * cur.x + cur.y * cur.y);
  const float Lc = max_prop(L, 1e-8f);
  const float stx = (cur.x / Lc) * (L - L0), sty = (cur.y / Lc) * (L - L0);
  const float shx = (cur.x - tx) - stx, shy = (cur.y - ty) - sty;
  return make_float2(((stx + shx * d.k_shear) * d.k_stretch) * 0.5f, ((sty + shy * d.k_shear) * d.k_stretch) * 0.5f);
}

// IB point p in lattice units (fluid.py:236-263): node p's position times the grid scale,
// or with synthetic pairs (p < N: +, p >= N: -, node = p mod N) that point moved by
// width * perp * mean_scale, where perp is the normal of the chain tangent, the sum of the
// node's edge vectors in the reference's update order (src updates, then tgt updates),
// normalised by sqrt(|t|^2 + EPSIL).
__device__ __forceinline__ float2 ib_point(const RDesc& d, int p, int node, float x, float y) {
  const float gx = x * d.scale_x, gy = y * d.scale_y;
  if (!(d.syn_w > 0.0f)) return make_float2(gx, gy);
  float tx = 0.0f, ty = 0.0f;
  for (int j = d.ne_off[node]; j < d.ne_off[node + 1]; ++j) {
    const int e = d.ne_idx[j] >> 1;
    const int s = d.pairs[2 * e], g = d.pairs[2 * e + 1];
    const float2 ev = min_image(d.pos[2 * g], d.pos[2 * g + 1], d.pos[2 * s], d.pos[2 * s + 1], (float)d.W, (float)d.H);
    tx = tx + ev.x;
    ty = ty + ev.y;
  }
  const float nrm = sqrtf((tx * tx + ty * ty) + MC_EPSIL);
  const float ux = tx / nrm, uy = ty / nrm;
  const float ox = (d.syn_w * (-uy)) * d.syn_ms, oy = (d.syn_w * ux) * d.syn_ms;
  return p < d.N ? make_float2(gx + ox, gy + oy) : make_float2(gx - ox, gy - oy);
}

// Contribution k appended to its cell; true when it is the cell's first of this step.
__device__ __forceinline__ bool ib_append(const RDesc& d, int cell, int k) {
  const int pos = atomicAdd(d.ib_cnt + cell, 1);
  if (pos < d.ib_cap) {
    d.ib_bucket[(size_t)cell * d.ib_cap + pos] = k;
  } else {
    const int e = atomicAdd(d.ib_ctl, 1);
    d.ib_ovf[e] = k;
    d.ib_ovf_next[e] = atomicExch(d.ib_ovf_head + cell, e);
  }
  return pos == 0;
}

// Velocity (simulate.py:83-84), the IB point in lattice units (fluid.py:236-239) and its
// K x K stencil (fluid.py:40-79), its contributions appended to their cells, the cells' first
// ones making them touched cells; and the clearing of the node's CIC deposit cells (the deposit
// grid stays zero between steps).  One thread per IB point, any K.
__global__ void __launch_bounds__(256) k_stencil(const RDesc* __restrict__ D, const int* __restrict__ off, int n) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int p = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;  // IB point
  if (p >= d.NI) return;
  const int gi = p < d.N ? p : p - d.N;
  const float x = d.pos[2 * gi], y = d.pos[2 * gi + 1];
  const float vx = (x - d.prev[2 * gi]) / d.dt, vy = (y - d.prev[2 * gi + 1]) / d.dt;
  if (p < d.N) {
    d.vel[2 * gi] = vx;
    d.vel[2 * gi + 1] = vy;
    if (d.enable_steric) {
#pragma unroll
      for (int c = 0; c < 4; ++c) d.dep[d.c_cell[c * d.N + gi]] = 0.0f;
    }
  }
  if (!d.enable_fluid) return;
  const int K = d.K, K2 = K * K;
  const float2 gp = ib_point(d, p, gi, x, y);
  const float gx = gp.x, gy = gp.y;
  d.nvl[p] = make_float2((vx * d.scale_x) * d.dt, (vy * d.scale_y) * d.dt);
  const int half = (K - 1) / 2;
  const float hw = (float)K / 2.0f;
  const float sx = floorf(gx) - (float)half, sy = floorf(gy) - (float)half;
  float wx[8], wy[8];
  int cx[8], cy[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    if (a < K) {
      const float rx = fabsf((sx + (float)a) - gx) / hw;
      const float ry = fabsf((sy + (float)a) - gy) / hw;
      wx[a] = rx <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * rx) / 2.0f)) : 0.0f;
      wy[a] = ry <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * ry) / 2.0f)) : 0.0f;
      cx[a] = imod_floor((int)(sx + (float)a), d.lW);
      cy[a] = imod_floor((int)(sy + (float)a), d.lH);
    }
  }
  float sum = 0.0f;
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if (a < K && b < K) sum = sum + wx[a] * wy[b];
  const float den = sum + MC_EPSIL;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    if (a < K) {
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        if (b < K) {
          const int k = p * K2 + a * K + b, cell = cy[b] * d.lW + cx[a];
          d.ib_w[k] = (wx[a] * wy[b]) / den;
          if (ib_append(d, cell, k) && !d.ib_list) d.h_new[atomicAdd(d.ib_ctl + 2, 1)] = cell;
        }
      }
    }
  }
}

// The same work for K <= 4 with 4 lanes per IB point, lane a a column of the stencil: two cosines
// and up to four contributions per lane.  The weights' sum is taken in entry order a * K + b by
// every lane, so the result equals the one-thread-per-point kernel's.  The touched cells of a warp
// (8 consecutive points) are numbered together, so that neighbours on a rod stay neighbours in the
// list of touched cells.  Bound by the latency of the atomics.  Before, 16 lanes per point computed
// all cosines 4 times over and took slots in 16x16 tiles: a batch of 64
// uneven rollouts with 74 k points 39 -> 23 us per launch, 1024^2 with 16,384 points 8.8 -> 9.2 us
// (latency on both sides; the kernel that follows gains more).
__global__ void __launch_bounds__(128) k_stencil4(const RDesc* __restrict__ D, const int* __restrict__ off, int n) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const int t = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  const int NI = d.NI, N = d.N;
  const int p = min(t >> 2, NI - 1), a = t & 3, lane = threadIdx.x & 31;
  const bool on = (t >> 2) < NI;
  const int gi = p < N ? p : p - N;
  // the predecessor (k_chain or k_node, without rods k_steric) writes positions and angles only
  const float2 pv = __ldcg(reinterpret_cast<const float2*>(d.prev) + gi);
  int dep = -1;
  if (on && p < N && d.enable_steric) dep = __ldcg(d.c_cell + a * N + gi);
  after_previous();
  const float x = d.pos[2 * gi], y = d.pos[2 * gi + 1];
  const float vx = (x - pv.x) / d.dt, vy = (y - pv.y) / d.dt;
  if (on && p < N) {
    if (a == 0) {
      d.vel[2 * gi] = vx;
      d.vel[2 * gi + 1] = vy;
    }
    if (dep >= 0) d.dep[dep] = 0.0f;
  }
  if (!d.enable_fluid) return;
  const int K = d.K;
  const float2 g = ib_point(d, p, gi, x, y);
  if (on && a == 0) d.nvl[p] = make_float2((vx * d.scale_x) * d.dt, (vy * d.scale_y) * d.dt);
  const float half = (float)((K - 1) / 2), hw = (float)K / 2.0f;
  const float bx = (floorf(g.x) - half) + (float)a, by = (floorf(g.y) - half) + (float)a;
  const float rx = fabsf(bx - g.x) / hw, ry = fabsf(by - g.y) / hw;
  const float wxa = rx <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * rx) / 2.0f)) : 0.0f;
  const float wya = ry <= 2.0f ? 0.25f * (1.0f + cosf((MC_PI_F * ry) / 2.0f)) : 0.0f;
  const int cx = imod_floor((int)bx, d.lW), cya = imod_floor((int)by, d.lH) * d.lW;
  const unsigned full = 0xffffffffu;
  float w[4];
  int cell[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    w[b] = wxa * __shfl_sync(full, wya, b, 4);
    cell[b] = __shfl_sync(full, cya, b, 4) + cx;
  }
  float sum = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float we = __shfl_sync(full, w[b], e, 4);
      if (e < K && b < K) sum = sum + we;
    }
  const float den = sum + MC_EPSIL;
  const bool mine = on && a < K;
  const int k0 = (p * K + a) * K;
  int pos[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) pos[b] = mine && b < K ? atomicAdd(d.ib_cnt + cell[b], 1) : -1;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (mine && b < K) d.ib_w[k0 + b] = w[b] / den;
  if (!d.ib_list) {
    int fresh = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) fresh += pos[b] == 0 ? 1 : 0;
    int before = fresh;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(full, before, o);
      if (lane >= o) before += v;
    }
    int base = 0;
    if (lane == 31 && before > 0) base = atomicAdd(d.ib_ctl + 2, before);
    base = __shfl_sync(full, base, 31) + before - fresh;
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (pos[b] == 0) d.h_new[base++] = cell[b];
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    if (pos[b] >= 0 && pos[b] < d.ib_cap) {
      d.ib_bucket[(size_t)cell[b] * d.ib_cap + pos[b]] = k0 + b;
    } else if (pos[b] >= 0) {
      const int e = atomicAdd(d.ib_ctl, 1);
      d.ib_ovf[e] = k0 + b;
      d.ib_ovf_next[e] = atomicExch(d.ib_ovf_head + cell[b], e);
    }
  }
}

// The prediction displaced by the steric force (simulate.py:55-65), written to the node positions
// the rod kernels start from.  The force (compute_field_steric_force_corrected, forces.py:41-81):
// -grad V by central differences of bilinear samples (map_coordinates order=1, mode="wrap",
// forces.py:30-34), minus the analytic Gaussian of global neighbours gi-n..gi+n (the 0 <= j < N
// mask only, as in the reference).
//
// 4 lanes per node: lane q takes one of the four samples and every fourth neighbour, whose terms
// are added in neighbour order.  Bound by latency; the neighbours do not need the field, so their
// part is done while the predecessor drains (the filter's last pass, which writes the field alone; pred
// and predw are k_predict's, three kernels before).
__global__ void __launch_bounds__(128) k_steric(const RDesc* __restrict__ D, const int* __restrict__ off, int n) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const int t = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  const int gi = min(t >> 2, d.N - 1), q = t & 3;
  if (!d.enable_steric) {
    after_previous();
    if ((t >> 2) < d.N && q < 2) d.pos[2 * gi + q] = d.pred[2 * gi + q];
    return;
  }
  const unsigned full = 0xffffffffu;
  const float2* predw = reinterpret_cast<const float2*>(d.predw);
  const float W = (float)d.W, H = (float)d.H;
  const float2 p = __ldcg(predw + gi);
  float2 x = __ldcg(reinterpret_cast<const float2*>(d.pred) + gi);
  const int nsk = d.st_skip;
  float ax = 0.0f, ay = 0.0f;
  for (int o0 = -nsk; o0 <= nsk; o0 += 4) {
    float tx = 0.0f, ty = 0.0f;
    if (o0 + q <= nsk) {
      const int j = gi + o0 + q;
      const float valid = (j >= 0 && j < d.N) ? 1.0f : 0.0f;
      const float2 pj = __ldcg(predw + (j < 0 ? 0 : (j >= d.N ? d.N - 1 : j)));
      const float2 rr = min_image(p.x, p.y, pj.x, pj.y, W, H);
      const float d2 = rr.x * rr.x + rr.y * rr.y;
      const float K = expf(-d2 / d.st_2s2) / d.st_norm;
      const float kv = K * valid;
      tx = kv * rr.x;
      ty = kv * rr.y;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ax = ax + __shfl_sync(full, tx, k, 4);
      ay = ay + __shfl_sync(full, ty, k, 4);
    }
  }
  // sample q: +x, -x, +y, -y by half a cell
  const float e = (q & 1) ? -0.5f : 0.5f;
  const float xx = q < 2 ? p.x + e : p.x, yy = q < 2 ? p.y : p.y + e;
  const float ly = floorf(yy), lx = floorf(xx);
  const float sy = yy - ly, sx = xx - lx;
  const float wy0 = 1.0f - sy, wx0 = 1.0f - sx;
  const int iy = (int)ly, ix = (int)lx;
  const int ix0 = imod_floor(ix, d.W), ix1 = imod_floor(ix + 1, d.W);
  const float* V0 = d.steric + (size_t)imod_floor(iy, d.H) * d.W;
  const float* V1 = d.steric + (size_t)imod_floor(iy + 1, d.H) * d.W;
  after_previous();
  float v = (wy0 * wx0) * V0[ix0];
  v = v + (wy0 * sx) * V0[ix1];
  v = v + (sy * wx0) * V1[ix0];
  v = v + (sy * sx) * V1[ix1];
  const float vxp = __shfl_sync(full, v, 0, 4), vxm = __shfl_sync(full, v, 1, 4);
  const float vyp = __shfl_sync(full, v, 2, 4), vym = __shfl_sync(full, v, 3, 4);
  float fx = -((vxp - vxm) / 1.0f), fy = -((vyp - vym) / 1.0f);
  if (nsk > 0) {
    fx = fx - d.st_coef * ax;
    fy = fy - d.st_coef * ay;
  }
  x.x = x.x + (fx * d.st_strength) * d.dt;
  x.y = x.y + (fy * d.st_strength) * d.dt;
  if ((t >> 2) < d.N && q == 0) {  // the caller's buffer: no alignment beyond a float's
    d.pos[2 * gi] = x.x;
    d.pos[2 * gi + 1] = x.y;
  }
}

// ---------------------------------------------------------------- chains: CTA per rod
// One CTA (one team) per chain rod; S: the longest chain of the plan.  At least four warps where all
// CTAs run at once (kChainFill: 6 of 4 warps of 80 registers on each of 148 SMs), so that the sines
// and cosines of a short rod's iterations do not fall to a single warp; beyond, issue slots are what
// is short, and a rod takes the warps that its nodes need.  Per launch with 4 warps and with the rod's
// own, rods of 32 nodes: 512 12.8 and 14.8 us, 888 14.8 and 14.7, 1,500 22.7 and 16.7, 8,000 78 and 39
// (one warp per rod with all phases in one loop: 17, 19, 18.6 and 43); of 64: 888 19.0 and 18.9, 4,000
// 62 and 56 (27 and 42: two nodes per lane need no ghosts, which count once the SMs are full).
constexpr int kChainFill = 6 * 148;
__global__ void __launch_bounds__(384) k_chain(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                               const int* tdev, int S) {
  extern __shared__ float2 chain_tab[];
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const TeamOf<1> tm = {(int)threadIdx.x >> 5, (int)blockDim.x >> 5, 1};
  chain_rod<true>(d, d.chain_info[blockIdx.x - off[r]], __ldcg(tdev), tm, d.pos, chain_tab, S);
}

// ---------------------------------------------------------------- general rods: CTA per rod
__global__ void k_node(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                       const int* tdev) {
  extern __shared__ float sm[];
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int comp = d.generic_comp[blockIdx.x - off[r]];
  const int n0 = d.comp_n[comp], nn = d.comp_n[comp + 1] - n0;
  const int e0 = d.comp_e[comp], ne = d.comp_e[comp + 1] - e0;
  const int b0 = d.comp_b[comp], nb = d.comp_b[comp + 1] - b0;
  float* px = sm;
  float* py = px + d.max_comp_nodes;
  float* th = py + d.max_comp_nodes;
  float* l0 = th + d.max_comp_edges;
  float* fx = l0 + d.max_comp_edges;
  float* fy = fx + d.max_comp_edges;
  float* corr = fy + d.max_comp_edges;
  float* ra = corr + d.max_comp_pairs;
  float* kb = ra + d.max_comp_pairs;
  const int tid = threadIdx.x, bd = blockDim.x;
  const int t = *tdev;

  for (int b = tid; b < nb; b += bd) {
    ra[b] = rest_angle(d, b0 + b, t);
    kb[b] = d.kb[b0 + b];
  }
  for (int e = tid; e < ne; e += bd) {
    th[e] = d.theta[e0 + e];
    l0[e] = d.rest_len[e0 + e];
  }
  for (int i = tid; i < nn; i += bd) {
    px[i] = d.pos[2 * (n0 + i)];
    py[i] = d.pos[2 * (n0 + i) + 1];
  }
  __syncthreads();

  const bool cosserat = d.solver == 1;
  for (int it = 0; it < d.cycles; ++it) {
    // theta pass over bending pairs (pbd.py:23-49; stable_cosserat.py:55-82)
    for (int b = tid; b < nb; b += bd) {
      const int ein = d.bpairs[2 * (b0 + b)] - e0, eout = d.bpairs[2 * (b0 + b) + 1] - e0;
      corr[b] = bend_corr(th[ein], th[eout], ra[b], kb[b]);
    }
    __syncthreads();
    for (int e = tid; e < ne; e += bd) {
      const int ge = e0 + e;
      float acc = 0.0f;
      for (int j = d.ep_off[ge]; j < d.ep_off[ge + 1]; ++j) {
        const int code = d.ep_idx[j];
        const float c = corr[(code >> 1) - b0];
        acc = (code & 1) ? acc + (-c) : acc + c;
      }
      if (cosserat) {
        const int s = d.pairs[2 * ge] - n0, g = d.pairs[2 * ge + 1] - n0;
        const float2 r = min_image(px[g], py[g], px[s], py[s], (float)d.W, (float)d.H);
        th[e] = cos_pull(th[e] + acc / d.edeg[ge], r.x, r.y);
      } else {
        th[e] = th[e] + (acc / d.edeg[ge]) * 1.8f;
      }
    }
    __syncthreads();
    // position pass over edges (pbd.py:51-89; stable_cosserat.py:84-119)
    for (int e = tid; e < ne; e += bd) {
      const int s = d.pairs[2 * (e0 + e)] - n0, g = d.pairs[2 * (e0 + e) + 1] - n0;
      if (cosserat) {
        const float2 r = min_image(px[g], py[g], px[s], py[s], (float)d.W, (float)d.H);
        float sn, cs;
        sincosf(th[e], &sn, &cs);
        const float kl = d.k_stretch / l0[e];
        fx[e] = kl * (r.x / l0[e] - cs);
        fy[e] = kl * (r.y / l0[e] - sn);
      } else {
        const float2 f = edge_force(d, th[e], l0[e], px[s], py[s], px[g], py[g]);
        fx[e] = f.x;
        fy[e] = f.y;
      }
    }
    __syncthreads();
    if (cosserat) {
      // implicit update with inertia: per node (w (y0 - x) + sum +-f_e) / (w + sum k_s/l_e^2),
      // y0 = the positions this kernel started from (still in global memory)
      const float w = d.cos_w;
      for (int i = tid; i < nn; i += bd) {
        const int gi = n0 + i;
        float ax = w * (d.pos[2 * gi] - px[i]), ay = w * (d.pos[2 * gi + 1] - py[i]), hh = w;
        for (int j = d.ne_off[gi]; j < d.ne_off[gi + 1]; ++j) {
          const int code = d.ne_idx[j];
          const int e = (code >> 1) - e0;
          if (code & 1) {
            ax = ax + (-fx[e]);
            ay = ay + (-fy[e]);
          } else {
            ax = ax + fx[e];
            ay = ay + fy[e];
          }
          hh = hh + d.k_stretch / (l0[e] * l0[e]);
        }
        px[i] = px[i] + ax / hh;
        py[i] = py[i] + ay / hh;
      }
      __syncthreads();
      continue;
    }
    for (int i = tid; i < nn; i += bd) {
      const int gi = n0 + i;
      float ax = 0.0f, ay = 0.0f;
      for (int j = d.ne_off[gi]; j < d.ne_off[gi + 1]; ++j) {
        const int code = d.ne_idx[j];
        const int e = (code >> 1) - e0;
        if (code & 1) {
          ax = ax + (-fx[e]);
          ay = ay + (-fy[e]);
        } else {
          ax = ax + fx[e];
          ay = ay + fy[e];
        }
      }
      const float dg = d.ndeg[gi];
      px[i] = px[i] + ax / dg;
      py[i] = py[i] + ay / dg;
    }
    __syncthreads();
  }

  for (int e = tid; e < ne; e += bd) d.theta[e0 + e] = th[e];
  for (int i = tid; i < nn; i += bd) {
    d.pos[2 * (n0 + i)] = px[i];
    d.pos[2 * (n0 + i) + 1] = py[i];
  }
}

void launch_predict(const Launch& L, int* tdev) { launch(L, k_predict, kNodeThreads, 0, L.d, L.off, L.n, tdev); }
void launch_steric(const Launch& L) { launch(L, k_steric, 128, 0, L.d, L.off, L.n); }
void launch_stencil(const Launch& L) { launch(L, k_stencil, kNodeThreads, 0, L.d, L.off, L.n); }
void launch_stencil4(const Launch& L) { launch(L, k_stencil4, 128, 0, L.d, L.off, L.n); }
void launch_node(const Launch& L, const int* tdev, size_t smem, int bs) {
  launch(L, k_node, bs, smem, L.d, L.off, L.n, tdev);
}
void launch_chain(const Launch& L, const int* tdev, int longest) {
  const int need = chain_warps(longest), warps = need < 4 && L.grid <= kChainFill ? 4 : need;
  launch(L, k_chain, 32 * warps, (size_t)chain_smem(longest) * sizeof(float2), L.d, L.off, L.n, tdev, longest);
}
cudaError_t node_set_smem(size_t bytes) {
  return cudaFuncSetAttribute(k_node, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace mc
