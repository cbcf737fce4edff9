// Chain rods (edge i = (node i, node i+1), pair i = (edge i, edge i+1)): the iterations of
// pbd_rod_constraint (src/microcosmos/solver/pbd.py:14-91) and stable_cosserat_constraint
// (src/microcosmos/solver/stable_cosserat.py:13-119) for one rod by a team of warps.
//
// One node (and edge and pair) per lane.  What bounds it is the length of one rod's chain of
// dependent operations, not the amount of work, so the chain is cut where the equations allow:
//  * the PBD angle pass reads no position, so all iterations' angles are advanced first (about
//    175 cycles each) and kept in shared memory; the sines and cosines of every (iteration,
//    edge) are then independent and spread over all threads of the team; the position pass
//    reads the finished rest vectors.  One lane's chain per iteration no longer holds the angle
//    update and the sincos;
//  * rods of more than 32 nodes use several warps instead of several nodes per lane: each warp
//    owns kSegOwn nodes and carries kSegGhost more on each side, advanced redundantly, so that
//    warps exchange boundary values (one barrier) only every kSegGhost iterations (an angle or
//    position depends on its direct neighbours only).
// Measured (one B200, 20 iterations, per launch inside a rollout's graph): 256 64-node rods 22.6 ->
// 11.4 us, 1,032 rods of 16 to 128 nodes 56 -> 29.4 us; before: one warp per rod with 2 or 4 nodes
// per lane, all phases in one loop.
#pragma once
#include "lbm_cell.cuh"

namespace mc {

constexpr int kSegOwn = 22;
constexpr int kSegGhost = 5;  // (the Cosserat passes: two nodes per iteration on the left, two iterations)
constexpr int kThetaChunk = 20;  // iterations whose angles are kept at a time

__host__ __device__ constexpr int chain_warps(int nn) { return nn <= 32 ? 1 : (nn + kSegOwn - 1) / kSegOwn; }
// shared memory of a team for rods of at most `S` nodes, in float2
__host__ __device__ constexpr int chain_smem(int S) { return (kThetaChunk + 2) * S; }

// The threads working on one rod.  All of them call chain_rod together; warps beyond the rod's
// own (chain_warps) help with the sines and cosines.
// BAR: the number of the team's barrier where it is known at compile time, else 0.  A barrier whose
// number is in a register makes the compiler reserve all 16 of a CTA, so that no more than 4 such CTAs
// fit on an SM (8,000 rods of 32 nodes in the chain kernel: 107 us per launch that way, 78 with 3
// barriers).
template <int BAR>
struct TeamOf {
  int warp, warps;  // this warp's index in the team, and the team's warps
  int bar;          // the team's named barrier; bar + 1 is that of a rod's own warps
  __device__ __forceinline__ void sync() const {
    if (warps == 1)
      __syncwarp();
    else if (BAR == 0)
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(warps * 32) : "memory");
    else
      asm volatile("bar.sync %0, %1;" ::"n"(BAR), "r"(warps * 32) : "memory");
  }
  // sync, and whether `p` holds for any thread of the team
  __device__ __forceinline__ bool sync_or(bool p) const {
    if (warps == 1) return __any_sync(0xffffffffu, p) != 0;
    int r;
    if (BAR == 0)
      asm volatile(
          "{\n\t.reg .pred a, b;\n\tsetp.ne.s32 a, %1, 0;\n\tbar.red.or.pred b, %2, %3, a;\n\t"
          "selp.s32 %0, 1, 0, b;\n\t}"
          : "=r"(r)
          : "r"((int)p), "r"(bar), "r"(warps * 32)
          : "memory");
    else
      asm volatile(
          "{\n\t.reg .pred a, b;\n\tsetp.ne.s32 a, %1, 0;\n\tbar.red.or.pred b, %2, %3, a;\n\t"
          "selp.s32 %0, 1, 0, b;\n\t}"
          : "=r"(r)
          : "r"((int)p), "n"(BAR), "r"(warps * 32)
          : "memory");
    return r != 0;
  }
  // The first rw warps, those of a rod.  Their barrier's count changes from rod to rod, so the whole
  // team meets at its own in between.  (With numbers per team all warps of a team stay with its
  // barrier, since not every team has two.)
  __device__ __forceinline__ TeamOf<BAR ? BAR + 1 : 0> rod(int rw) const {
    return {warp, rw, BAR ? BAR + 1 : rw == warps ? bar : bar + 1};
  }
};
using Team = TeamOf<0>;

// max that propagates NaN, for the range checks of the fast passes
__device__ __forceinline__ float max_track(float m, float v) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(v)));
  return r;
}
__device__ __forceinline__ float min_track(float m, float v) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(v));
  return r;
}

// fmod_floor of x = d + y / 2 where |d| < 1.49 y: x lies in (-y, 2 y), so one period at most is
// added or taken away (exactly).
constexpr float kNear = 1.49f;
__device__ __forceinline__ float fmod_near(float x, float y) {
  const float r = (x >= y) ? x - y : x;
  return (x < 0.0f) ? x + y : r;
}

// Length L and direction v / L of a segment with squared length s, each correctly rounded, without
// branches, by Newton and residual corrections of the hardware's approximations (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34, 1990): for the square root, g ~ sqrt(s) and h ~ 1 / (2 sqrt(s)) are refined together and
// the exact residual s - g g corrects g; for a quotient, with r = RN(1 / L), two corrections by
// the exact residual v - L q.  The root equals sqrtf for every float from 2^-50 to 2^38 and r equals
// 1 / L for every significand (tests/rod_arithmetic.cu compares them, and quotients and whole rods
// with the general path).  The bounds: s >= 2^-50, where the reference's floor of the length (1e-8)
// does not act either; components are min-image differences, so multiples of 2^-23, and at most
// half a domain's side, so that s stays far below 2^38.  A zero component may lose its sign, which
// no later sum can show.
constexpr float kNearLength2 = 0x1p-50f;
__device__ __forceinline__ float2 unit_near(float2 v, float s, float& L) {
  float y, r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
  float g = s * y, h = 0.5f * y;
  const float c = __fmaf_rn(-g, h, 0.5f);
  g = __fmaf_rn(g, c, g);
  h = __fmaf_rn(h, c, h);
  L = __fmaf_rn(__fmaf_rn(-g, g, s), h, g);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(L));
  r = __fmaf_rn(__fmaf_rn(-L, r, 1.0f), r, r);
  float qx = v.x * r, qy = v.y * r;
  qx = __fmaf_rn(__fmaf_rn(-L, qx, v.x), r, qx);
  qy = __fmaf_rn(__fmaf_rn(-L, qy, v.y), r, qy);
  qx = __fmaf_rn(__fmaf_rn(-L, qx, v.x), r, qx);
  qy = __fmaf_rn(__fmaf_rn(-L, qy, v.y), r, qy);
  return make_float2(qx, qy);
}

// Rest angle of pair gb at step t (the caller-side curvature actuation, if any); `store` keeps
// it in the state.
__device__ __forceinline__ float rest_angle(const RDesc& d, int gb, int t, bool store = true) {
  if (!d.act_amp) return __ldcg(d.rest_ang + gb);
  const float arg = d.act_omega[gb] * (float)(d.act_t0 + t) + d.act_phase[gb];
  const float a = d.act_c[gb] + d.act_amp[gb] * sinf(arg);
  if (store) d.rest_ang[gb] = a;
  return a;
}

// One theta correction (pbd.py:35-40).
__device__ __forceinline__ float bend_corr(float th_in, float th_out, float rest, float kb) {
  float diff = th_out - th_in;
  diff = fmod_floor(diff + MC_PI_F, MC_2PI_F) - MC_PI_F;
  return ((diff - rest) * kb) * 0.5f;
}

// One lane's place on its rod.
struct RodLane {
  int j, nn, ne, nb;  // node, edge and pair j of a rod of nn nodes (lanes off the rod: j < 0 or j >= nn)
  bool own;           // the node is this warp's own and not a neighbour's
};

// q angle passes (pbd.py:23-49); row k of tab keeps the angles after pass k.  NEAR: without the
// slow path of the floored modulo; returns whether this lane would have needed it.
template <bool NEAR, bool SEVERAL, class T>
__device__ __forceinline__ bool theta_passes(const T& rod, const RodLane& l, int q, float& th, float ra, float kb,
                                             float edg, float2* tab, int S) {
  const bool pair = l.j >= 0 && l.j < l.nb, prev = l.j >= 1 && l.j - 1 < l.nb, edge = l.j >= 0 && l.j < l.ne;
  const bool keep = l.own && edge;
  float far = 0.0f;
  int left = kSegGhost;
  float2* row = tab + max(l.j, 0);
  for (int k = 0; k < q; ++k, row += S) {
    if (SEVERAL) {
      if (left == 0) {
        rod.sync();
        if (!l.own && edge) th = (row - S)->x;
        left = kSegGhost;
      }
      --left;
    }
    const float nx = __shfl_down_sync(0xffffffffu, th, 1);
    float c;
    if (NEAR) {
      const float d = nx - th;
      far = max_track(far, d);
      c = (((fmod_near(d + MC_PI_F, MC_2PI_F) - MC_PI_F) - ra) * kb) * 0.5f;
    } else {
      c = bend_corr(th, nx, ra, kb);
    }
    // the terms that do not exist are zeros
    c = pair ? c : 0.0f;
    float pv = __shfl_up_sync(0xffffffffu, c, 1);
    pv = prev ? pv : 0.0f;
    th = th + ((c - pv) * edg) * 1.8f;
    if (keep) row->x = th;
  }
  return NEAR && pair && l.own && !(far < kNear * MC_2PI_F);
}

// q position passes (pbd.py:51-89) with the rest vectors in tab; first: no pass came before them.
// NEAR: without the slow paths of the modulo, the square root and the divisions.
template <bool NEAR, bool SEVERAL, class T>
__device__ __forceinline__ bool position_passes(const T& rod, const RodLane& l, int q, bool first, float& x,
                                                float& y, float l0, float ndg, float Wf, float Hf, float ksh,
                                                float kst, const float2* tab, float2* ex, int& buf, int S) {
  // (lane 31 of a warp sees no next node: with several warps its edge is a neighbour's)
  const bool node = l.j >= 0 && l.j < l.nn, prev = l.j >= 1;
  const bool edge = l.j >= 0 && l.j < l.ne && (threadIdx.x & 31) < 31;
  const float hx = Wf / 2.0f, hy = Hf / 2.0f;
  float far_x = 0.0f, far_y = 0.0f, s_min = 1.0f;
  int left = first ? kSegGhost : 0;
  const float2* row = tab + min(max(l.j, 0), max(l.ne - 1, 0));
  for (int k = 0; k < q; ++k, row += S) {
    if (SEVERAL) {
      if (left == 0) {
        if (l.own) ex[buf * S + l.j] = make_float2(x, y);
        rod.sync();
        if (!l.own && node) {
          const float2 p = ex[buf * S + l.j];
          x = p.x;
          y = p.y;
        }
        buf ^= 1;
        left = kSegGhost;
      }
      --left;
    }
    const float2 tv = *row;
    const float xn = __shfl_down_sync(0xffffffffu, x, 1), yn = __shfl_down_sync(0xffffffffu, y, 1);
    float2 cur, dir;
    float L;
    if (NEAR) {
      const float dx = xn - x, dy = yn - y;
      cur.x = fmod_near(dx + hx, Wf) - hx;
      cur.y = fmod_near(dy + hy, Hf) - hy;
      const float s = cur.x * cur.x + cur.y * cur.y;
      dir = unit_near(cur, s, L);
      far_x = max_track(far_x, dx);
      far_y = max_track(far_y, dy);
      s_min = min_track(s_min, s);
    } else {
      cur = min_image(xn, yn, x, y, Wf, Hf);
      L = sqrtf(cur.x * cur.x + cur.y * cur.y);
      const float Lc = max_prop(L, 1e-8f);
      dir = make_float2(cur.x / Lc, cur.y / Lc);
    }
    const float stx = dir.x * (L - l0), sty = dir.y * (L - l0);
    const float shx = (cur.x - tv.x) - stx, shy = (cur.y - tv.y) - sty;
    const float fx = edge ? ((stx + shx * ksh) * kst) * 0.5f : 0.0f;
    const float fy = edge ? ((sty + shy * ksh) * kst) * 0.5f : 0.0f;
    float fxp = __shfl_up_sync(0xffffffffu, fx, 1), fyp = __shfl_up_sync(0xffffffffu, fy, 1);
    fxp = prev ? fxp : 0.0f;
    fyp = prev ? fyp : 0.0f;
    x = x + (fx - fxp) * ndg;
    y = y + (fy - fyp) * ndg;
  }
  return NEAR && edge && l.own && !(far_x < kNear * Wf && far_y < kNear * Hf && s_min >= kNearLength2);
}

// All iterations of a PBD rod of rw warps.  The passes run without the slow paths of the modulo
// and the divisions first (their branches would lie on the dependent chain); if any lane needed
// one, the chunk is done again from its start with them.  start() gives the positions; the first
// chunk's angles and rest vectors do not need them.
template <bool SEVERAL, class F, class T>
__device__ __forceinline__ void pbd_iterations(const F& start, const RDesc& d, const T& tm, int rw, const RodLane& l, int e0,
                                               float& x, float& y, float& th, float l0, float ra, float kb, float edg,
                                               float ndg, float2* tab, int S) {
  const int lane = threadIdx.x & 31;
  const bool act = tm.warp < rw, edge = l.j >= 0 && l.j < l.ne;
  const float Wf = (float)d.W, Hf = (float)d.H, ksh = d.k_shear, kst = d.k_stretch;
  float2* ex = tab + kThetaChunk * S;
  const auto rod = tm.rod(rw);
  const int cycles = d.cycles;
  int buf = 0;
  if (cycles <= 0) start();
  for (int it0 = 0; it0 < cycles; it0 += kThetaChunk) {
    const int q = min(kThetaChunk, cycles - it0);
    const float th0 = th;
    bool bad = false;
    if (act) bad = theta_passes<true, SEVERAL>(rod, l, q, th, ra, kb, edg, tab, S);
    if (tm.sync_or(bad)) {
      th = th0;
      if (act) theta_passes<false, SEVERAL>(rod, l, q, th, ra, kb, edg, tab, S);
      tm.sync();
    }
    if (SEVERAL) {
      if (act && !l.own && edge) th = tab[(q - 1) * S + l.j].x;
      tm.sync();
    }
    // rest vectors l0 (cos, sin) of every (iteration, edge): one iteration per warp at a time
    for (int e = lane; e < l.ne; e += 32) {
      const float le = d.rest_len[e0 + e];
#pragma unroll 2
      for (int k = tm.warp; k < q; k += tm.warps) {
        float sn, cs;
        sincosf(tab[k * S + e].x, &sn, &cs);
        tab[k * S + e] = make_float2(cs * le, sn * le);
      }
    }
    tm.sync();
    if (it0 == 0) start();
    const float x0 = x, y0 = y;
    const int buf0 = buf;
    bad = false;
    if (act)
      bad = position_passes<true, SEVERAL>(rod, l, q, it0 == 0, x, y, l0, ndg, Wf, Hf, ksh, kst, tab, ex, buf, S);
    if (tm.sync_or(bad)) {
      x = x0;
      y = y0;
      buf = buf0;
      if (act) position_passes<false, SEVERAL>(rod, l, q, it0 == 0, x, y, l0, ndg, Wf, Hf, ksh, kst, tab, ex, buf, S);
      tm.sync();
    }
  }
}

// a / b, correctly rounded, from r = RN(1 / b) and two corrections by the exact residual (see
// unit_near); a zero or between 2^-80 and 2^80, b between 2^-30 and 2^30.
__device__ __forceinline__ float div_near(float a, float b, float r) {
  float q = a * r;
  q = __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
  return __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
}
__device__ __forceinline__ float reciprocal(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return __fmaf_rn(__fmaf_rn(-b, r, 1.0f), r, r);
}

// Stable-Cosserat iterations of one rod (solver/stable_cosserat.py:13-119).  Phase 1: the bending
// pass without over-relaxation, then theta += wrap(atan2(r) - theta) * 0.05 with r the segment's
// min-image vector.  Phase 2: x += (w (y0 - x) + f_j - f_{j-1}) / ((w + H_j) + H_{j-1}), f =
// (k_s/l)(r/l - d), H = k_s/l^2, y0 the inertial prediction (the positions the rod started from).
// The angles depend on the positions here, so the two phases alternate; values travel two nodes
// to the right per iteration, so the warps exchange after every second one.  The divisors do not
// change, so NEAR divides by their reciprocals (div_near); it returns whether this lane left the
// range where that and the one-period modulo are exact.
template <bool NEAR, bool SEVERAL, class T>
__device__ __forceinline__ bool cosserat_iterations(const RDesc& d, const T& rod, const RodLane& l, float& x,
                                                    float& y, float& th, float l0, float ra, float kb, float edg,
                                                    float2* ex, float* ext, int S) {
  const int j = l.j;
  const bool node = j >= 0 && j < l.nn, pair = j >= 0 && j < l.nb, pair_prev = j >= 1 && j - 1 < l.nb, prev = j >= 1;
  const bool edge = j >= 0 && j < l.ne && (threadIdx.x & 31) < 31;
  const float W = (float)d.W, H = (float)d.H, hx = W / 2.0f, hy = H / 2.0f;
  const float w = d.cos_w, x0 = x, y0 = y;
  const float le = edge ? l0 : 1.0f;
  const float kl = edge ? d.k_stretch / le : 0.0f, he = edge ? d.k_stretch / (le * le) : 0.0f;
  const float hep = __shfl_up_sync(0xffffffffu, he, 1);
  float hh = w;
  if (j < l.ne) hh = hh + he;
  if (prev) hh = hh + hep;
  const float rl = NEAR ? reciprocal(le) : 0.0f, rh = NEAR ? reciprocal(hh) : 0.0f;
  float far_t = 0.0f, far_x = 0.0f, far_y = 0.0f, big = 0.0f, small = 1.0f;
  int buf = 0, left = 2;
  for (int it = 0; it < d.cycles; ++it) {
    if (SEVERAL) {
      if (left == 0) {
        if (l.own) {
          ex[buf * S + j] = make_float2(x, y);
          ext[buf * S + j] = th;
        }
        rod.sync();
        if (!l.own && node) {
          const float2 p = ex[buf * S + j];
          x = p.x;
          y = p.y;
          th = ext[buf * S + j];
        }
        buf ^= 1;
        left = 2;
      }
      --left;
    }
    const float nx = __shfl_down_sync(0xffffffffu, th, 1);
    const float xn = __shfl_down_sync(0xffffffffu, x, 1), yn = __shfl_down_sync(0xffffffffu, y, 1);
    float c;
    float2 r;
    if (NEAR) {
      const float dt = nx - th, dx = xn - x, dy = yn - y;
      far_t = pair ? max_track(far_t, dt) : far_t;
      far_x = max_track(far_x, dx);
      far_y = max_track(far_y, dy);
      c = (((fmod_near(dt + MC_PI_F, MC_2PI_F) - MC_PI_F) - ra) * kb) * 0.5f;
      r = make_float2(fmod_near(dx + hx, W) - hx, fmod_near(dy + hy, H) - hy);
    } else {
      c = bend_corr(th, nx, ra, kb);
      r = min_image(xn, yn, x, y, W, H);
    }
    // lanes without an edge take a unit segment, off the slow paths of atan2
    if (!edge) r = make_float2(1.0f, 1.0f);
    c = pair ? c : 0.0f;
    float pv = __shfl_up_sync(0xffffffffu, c, 1);
    pv = pair_prev ? pv : 0.0f;
    th = th + (c - pv) * edg;
    if (NEAR) {
      const float a = atan2f(r.y, r.x) - th;
      far_t = max_track(far_t, edge ? a : 0.0f);
      th = th + (fmod_near(a + MC_PI_F, MC_2PI_F) - MC_PI_F) * 0.05f;
    } else {
      th = cos_pull(th, r.x, r.y);
    }
    float sn, cs;
    sincosf(th, &sn, &cs);
    const float qx = NEAR ? div_near(r.x, le, rl) : r.x / le, qy = NEAR ? div_near(r.y, le, rl) : r.y / le;
    const float fx = edge ? kl * (qx - cs) : 0.0f, fy = edge ? kl * (qy - sn) : 0.0f;
    float fxp = __shfl_up_sync(0xffffffffu, fx, 1), fyp = __shfl_up_sync(0xffffffffu, fy, 1);
    fxp = prev ? fxp : 0.0f;
    fyp = prev ? fyp : 0.0f;
    const float ax = (w * (x0 - x) + fx) - fxp, ay = (w * (y0 - y) + fy) - fyp;
    if (NEAR) {
      big = max_track(max_track(big, ax), ay);
      small = min_track(min_track(small, ax == 0.0f ? 1.0f : fabsf(ax)), ay == 0.0f ? 1.0f : fabsf(ay));
      x = x + div_near(ax, hh, rh);
      y = y + div_near(ay, hh, rh);
    } else {
      x = x + ax / hh;
      y = y + ay / hh;
    }
  }
  if (!NEAR || !l.own) return false;
  const bool moves = !(big < 0x1p80f && small > 0x1p-80f && hh > 0x1p-30f && hh < 0x1p30f);
  const bool turns = edge && !(far_t < kNear * MC_2PI_F && far_x < kNear * W && far_y < kNear * H && le > 0x1p-30f &&
                               le < 0x1p30f);
  return moves || turns;
}

template <bool SEVERAL, class T>
__device__ __forceinline__ void cosserat_rod(const RDesc& d, const T& rod, const RodLane& l, float& x, float& y,
                                             float& th, float l0, float ra, float kb, float edg, float2* tab, int S) {
  float2* ex = tab + kThetaChunk * S;
  float* ext = reinterpret_cast<float*>(tab);
  const float xs = x, ys = y, ts = th;
  if (rod.sync_or(cosserat_iterations<true, SEVERAL>(d, rod, l, x, y, th, l0, ra, kb, edg, ex, ext, S))) {
    x = xs;
    y = ys;
    th = ts;
    cosserat_iterations<false, SEVERAL>(d, rod, l, x, y, th, l0, ra, kb, edg, ex, ext, S);
  }
}

// All cycles_per_step iterations at step t of the chain info = (first node, nodes, first edge, first
// pair).  pos: the rollout's node positions (x, y), updated in place; tab: chain_smem(S) float2 of
// shared memory, S >= the rod's nodes.  Every warp of the team calls it with the same arguments.  A PBD
// rod ends with a barrier of the whole team, a Cosserat rod does not: its exchange buffers and its own
// warps' barrier are free for another rod of the team only after one (k_node_step).
template <bool CHAINED, class T>
__device__ __forceinline__ void chain_rod(const RDesc& d, int4 info, int t, const T& tm, float* pos, float2* tab,
                                          int S) {
  const int lane = threadIdx.x & 31;
  const int n0 = info.x, nn = info.y, e0 = info.z, b0 = info.w;
  RodLane l;
  l.nn = nn;
  l.ne = nn - 1;
  l.nb = nn > 2 ? nn - 2 : 0;
  const int rw = chain_warps(nn);
  const bool several = rw > 1, act = tm.warp < rw;
  l.j = several ? tm.warp * kSegOwn + lane - kSegGhost : lane;
  l.own = act && l.j < nn && (!several || (lane >= kSegGhost && lane < kSegGhost + kSegOwn));
  const int j = l.j, ne = l.ne, nb = l.nb;
  float x = 0.0f, y = 0.0f, th = 0.0f, l0 = 0.0f, ra = 0.0f, kb = 0.0f;
  // CHAINED: the predecessor, k_steric, writes the positions and touches nothing else of a rod; what a
  // PBD rod does without them comes first (the step counter, the angles and their passes, the rest
  // angles read and, under actuation, written)
  auto start = [&] {
    if (CHAINED) after_previous();
    if (act && j >= 0 && j < nn) {
      x = pos[2 * (n0 + j)];
      y = pos[2 * (n0 + j) + 1];
    }
  };
  auto late = [&] {
    if (CHAINED) start();
  };
  if (!CHAINED || d.solver == 1) start();
  if (act && j >= 0) {
    if (j < ne) {
      th = __ldcg(d.theta + e0 + j);
      l0 = d.rest_len[e0 + j];
    }
    if (j < nb) {
      ra = rest_angle(d, b0 + j, t, l.own);
      kb = d.kb[b0 + j];
    }
  }
  // chain degrees are 1 or 2, so x / deg == x * (1 / deg) exactly
  const float edg = ((j < nb) + (j >= 1 && j - 1 < nb)) == 2 ? 0.5f : 1.0f;
  const float ndg = ((j < ne) + (j >= 1 && j - 1 < ne)) == 2 ? 0.5f : 1.0f;
  if (d.solver == 1) {
    const auto rod = tm.rod(rw);
    if (act && several)
      cosserat_rod<true>(d, rod, l, x, y, th, l0, ra, kb, edg, tab, S);
    else if (act)
      cosserat_rod<false>(d, rod, l, x, y, th, l0, ra, kb, edg, tab, S);
  }
  else if (several)
    pbd_iterations<true>(late, d, tm, rw, l, e0, x, y, th, l0, ra, kb, edg, ndg, tab, S);
  else
    pbd_iterations<false>(late, d, tm, rw, l, e0, x, y, th, l0, ra, kb, edg, ndg, tab, S);
  if (l.own) {
    if (j < ne) d.theta[e0 + j] = th;
    pos[2 * (n0 + j)] = x;
    pos[2 * (n0 + j) + 1] = y;
  }
}

}  // namespace mc
