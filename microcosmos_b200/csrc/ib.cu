// Immersed-boundary coupling (src/microcosmos/solver/fluid.py:202-386) and the deterministic
// scatter-adds: of the stencils' contributions to their cells, and of the steric cloud-in-cell
// deposit (src/microcosmos/forces.py:98-115).
//
// Scatter-adds are never done with float atomics: integer atomics collect the contributions of a
// cell in arrival order, then they are ordered by contribution index and summed one after another,
// the reference's in-order scatter-add, bit-reproducibly.  IB contributions (k = point*K*K + entry)
// are collected per cell (k_stencil4, k_stencil) and one thread per touched cell ("head") orders
// them (k_ib_heads); the rounds work on the compact list of heads instead of full (H, W) grids.
// CIC contributions (k = corner*N + node) are collected per 16x16-cell tile and one CTA per tile
// counting-sorts them by cell (k_bin_tiles).
#include "lbm_cell.cuh"

namespace mc {

struct BinView {
  const int* cell;
  const float* w;
  int* store;
  int* tcount;
  int* ovf;
  int* ctl;
  int cap;
  int count;
  int gw;      // width of the grid the cells index
  int ntx;     // bin tiles per row of that grid
  int ntiles;  // bin tiles of that grid
};

__device__ __forceinline__ BinView bin_view(const RDesc& d) {
  BinView v;
  v.cell = d.c_cell; v.w = d.c_w; v.store = d.c_store; v.tcount = d.c_tcount; v.ovf = d.c_ovf;
  v.ctl = d.c_ctl; v.cap = d.c_cap; v.count = d.enable_steric ? 4 * d.N : 0;
  v.gw = d.W; v.ntx = d.ntile_x; v.ntiles = d.ntile_x * d.ntile_y;
  return v;
}

__device__ __forceinline__ int tile_of(const BinView& v, int cell) {
  const int cy = cell / v.gw, cx = cell - cy * v.gw;
  return (cy / kBinTile) * v.ntx + cx / kBinTile;
}
__device__ __forceinline__ unsigned local_of(const BinView& v, int cell) {
  const int cy = cell / v.gw, cx = cell - cy * v.gw;
  return (unsigned)((cy % kBinTile) * kBinTile + (cx % kBinTile));
}

__device__ void bitonic_sort_smem(unsigned* s, int P) {
  for (int k = 2; k <= P; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned a = s[i], b = s[ixj];
          const bool up = (i & k) == 0;
          if ((a > b) == up) {
            s[i] = b;
            s[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

__device__ __forceinline__ int lower_bound_u(const unsigned* a, int len, unsigned key) {
  int lo = 0, hi = len;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Deposit of one touched cell whose contributions are run[0..len) in increasing k, read from
// global memory (spilled tiles only): the in-order sum (forces.py:98-115).
__device__ __forceinline__ void deposit_cell(const RDesc& d, const BinView& v, const int* run, int len) {
  const int k0 = run[0];
  float acc = v.w[k0];
  for (int j = 1; j < len; ++j) acc = acc + v.w[run[j]];
  d.dep[v.cell[k0]] = acc;
}

// One CTA on one bin tile: sort the tile's contributions by (cell, k) and reduce every
// touched cell's run.  Tiles of at most capS contributions are sorted in shared memory;
// larger ones take the global-arena path.  skeys: dynamic shared memory of 4 * capS words, capS <= the
// bin capacity of every rollout of the launch (a power of two).
__device__ __forceinline__ int pc(int c) { return c + (c >> 3); }

__device__ void tile_work(const RDesc& d, int t, unsigned* skeys, int capS) {
  const int kCapS = capS;
  const int kChunk = 4 * capS;  // keys per shared-memory chunk sort on the spill path
  // per-cell counters at padded slots pc(c) = c + c / 8: the scan below gives each lane 8
  // consecutive cells, and the padding puts the lanes' slots on distinct banks
  __shared__ int cnt[kBinTile * kBinTile + kBinTile * kBinTile / 8];
  __shared__ int cpos[kBinTile * kBinTile + kBinTile * kBinTile / 8];
  __shared__ int hpos[kBinTile * kBinTile + kBinTile * kBinTile / 8];  // rank of a touched cell among the tile's
  __shared__ int tlist[kBinTile * kBinTile];  // the touched cells, by rank
  __shared__ int s_spill, s_heads, s_fill;
  const BinView v = bin_view(d);
  if (v.count == 0) return;
  const int total = v.tcount[t];
  if (total == 0) return;
  const int tid = threadIdx.x;
  const int ntiles = v.ntiles;
  int* bin = v.store + (size_t)t * v.cap;

  // fast path: the whole tile sorted in shared memory (capacity capS <= the bin capacity)
  if (total <= min(v.cap, kCapS)) {
    // shared layout: [0, C) packed (cell, rank) | [C, 2C) k | [2C, 3C) sorted k | [3C, 4C) sorted w
    unsigned* lr = skeys;
    int* kin = reinterpret_cast<int*>(skeys + kCapS);
    int* kout = reinterpret_cast<int*>(skeys + 2 * kCapS);
    float* wout = reinterpret_cast<float*>(skeys + 3 * kCapS);
    for (int c = tid; c < kBinTile * kBinTile; c += blockDim.x) cnt[pc(c)] = 0;
    if (tid == 0) s_heads = 0;
    __syncthreads();
    // counting sort by local cell; positions inside a cell come from shared atomics
    // (arbitrary order), so each cell's run is then ordered by k
    for (int i = tid; i < total; i += blockDim.x) {
      const unsigned e = (unsigned)bin[i];  // (local cell << 24) | k
      const unsigned lc = e >> 24;
      const int k = (int)(e & 0xffffffu);
      const int pos = atomicAdd(cnt + pc(lc), 1);
      lr[i] = (lc << 24) | (unsigned)pos;
      kin[i] = k;
    }
    __syncthreads();
    // exclusive scan of the 256 cell counts (one warp, 8 per lane) and the head count
    if (tid < 32) {
      int loc[8];
      int sum = 0, nz = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        loc[q] = cnt[tid * 9 + q];  // pc(tid * 8 + q)
        sum += loc[q];
        nz += loc[q] > 0;
      }
      int incl = sum, inz = nz;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, incl, o);
        int z = __shfl_up_sync(0xffffffffu, inz, o);
        if (tid >= o) {
          incl += y;
          inz += z;
        }
      }
      int run = incl - sum, hrun = inz - nz;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        cpos[tid * 9 + q] = run;
        hpos[tid * 9 + q] = hrun;
        run += loc[q];
        hrun += loc[q] > 0;
      }
      if (tid == 31) s_heads = inz;
    }
    __syncthreads();
    // the touched cells listed by rank
    for (int c = tid; c < kBinTile * kBinTile; c += blockDim.x)
      if (cnt[pc(c)] > 0) tlist[hpos[pc(c)]] = c;
    for (int i = tid; i < total; i += blockDim.x) {
      const unsigned key = lr[i];
      const int lc = (int)(key >> 24), pos = (int)(key & 0xffffffu);
      const int k = kin[i];
      kout[cpos[pc(lc)] + pos] = k;
      wout[cpos[pc(lc)] + pos] = v.w[k];
    }
    __syncthreads();
    // one thread per touched cell: order its run by k (runs are short), then reduce it
    const int nheads = s_heads;
    for (int hi = tid; hi < nheads; hi += blockDim.x) {
      const int c = tlist[hi];
      const int len = cnt[pc(c)];
      int* rk = kout + cpos[pc(c)];
      float* rw = wout + cpos[pc(c)];
      for (int a = 1; a < len; ++a) {
        const int key = rk[a];
        const float kw = rw[a];
        int b = a - 1;
        while (b >= 0 && rk[b] > key) {
          rk[b + 1] = rk[b];
          rw[b + 1] = rw[b];
          --b;
        }
        rk[b + 1] = key;
        rw[b + 1] = kw;
      }
      float acc = rw[0];
      for (int j = 1; j < len; ++j) acc = acc + rw[j];
      d.dep[v.cell[rk[0]]] = acc;
    }
    if (tid == 0) v.tcount[t] = 0;
    return;
  }

  // Spilled tile: gather its bin and its overflow entries into a private arena region,
  // sort by (cell, k) with shared-memory chunk sorts and rank merges, then reduce.
  if (tid == 0) s_spill = atomicAdd(v.ctl + 1, 2 * total);
  __syncthreads();
  const int base = ntiles * v.cap + s_spill;
  unsigned* bufA = reinterpret_cast<unsigned*>(v.store) + base;
  unsigned* bufB = bufA + total;
  const int nbin = min(total, v.cap);
  for (int i = tid; i < nbin; i += blockDim.x) bufB[i] = (unsigned)bin[i];  // already (local << 24) | k
  if (tid == 0) s_fill = nbin;
  __syncthreads();
  if (total > v.cap) {
    // the overflow list is unordered: every thread scans a stride of it for this tile's
    // entries (their order is restored by the sort below)
    const int no = v.ctl[0];
    for (int i = tid; i < no; i += blockDim.x) {
      const int k = v.ovf[i];
      if (tile_of(v, v.cell[k]) == t) bufB[atomicAdd(&s_fill, 1)] = (local_of(v, v.cell[k]) << 24) | (unsigned)k;
    }
  }
  __syncthreads();
  const int m = total;
  for (int c0 = 0; c0 < m; c0 += kChunk) {
    const int len = min(kChunk, m - c0);
    int P = 1;
    while (P < len) P <<= 1;
    for (int i = tid; i < P; i += blockDim.x) skeys[i] = i < len ? bufB[c0 + i] : 0xffffffffu;
    __syncthreads();
    bitonic_sort_smem(skeys, P);
    for (int i = tid; i < len; i += blockDim.x) bufA[c0 + i] = skeys[i];
    __syncthreads();
  }
  unsigned* src = bufA;
  unsigned* dst = bufB;
  for (int wdt = kChunk; wdt < m; wdt <<= 1) {
    for (int i = tid; i < m; i += blockDim.x) {
      const int ps = (i / (2 * wdt)) * (2 * wdt);
      const int a_len = min(wdt, m - ps);
      const int b0 = ps + a_len;
      const int b_len = max(0, min(wdt, m - b0));
      const unsigned key = src[i];
      int pos;
      if (i < b0)
        pos = (i - ps) + lower_bound_u(src + b0, b_len, key);
      else
        pos = (i - b0) + lower_bound_u(src + ps, a_len, key);
      dst[ps + pos] = key;
    }
    __syncthreads();
    unsigned* tmp = src;
    src = dst;
    dst = tmp;
  }
  // runs are located on the sorted keys; their k values go to the other buffer
  const unsigned* keys = src;
  int* kv = reinterpret_cast<int*>(dst);
  for (int i = tid; i < m; i += blockDim.x) kv[i] = (int)(keys[i] & 0xffffffu);
  __syncthreads();
  for (int i = tid; i < m; i += blockDim.x) {
    const unsigned lc = keys[i] >> 24;
    if (i > 0 && (keys[i - 1] >> 24) == lc) continue;
    int len = 1;
    while (i + len < m && (keys[i + len] >> 24) == lc) ++len;
    deposit_cell(d, v, kv + i, len);
  }
  if (tid == 0) v.tcount[t] = 0;
}

// The bin tiles that received contributions this step, listed by the producers as
// (rollout, tile) pairs (most tiles of a large or batched grid are empty and never
// listed).  A grid of as many CTAs as the GPU holds at once takes the listed tiles one at
// a time from a cursor (wl_count[2], reset with the list), so that no CTA is launched only
// to find nothing to do and uneven tiles balance across the CTAs.
__global__ void __launch_bounds__(256) k_bin_tiles(const RDesc* __restrict__ D, const int2* wl, int* wl_count,
                                                   int capS) {
  extern __shared__ unsigned dyn[];
  __shared__ int s_item;
  after_previous();
  const int count = *wl_count;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(wl_count + 2, 1);
    __syncthreads();
    const int i = s_item;
    if (i >= count) break;  // uniform across the CTA
    const int2 item = wl[i];
    tile_work(D[item.x], item.y, dyn, capS);
    __syncthreads();  // the shared arrays and s_item are reused by the next item
  }
}

// ---------------------------------------------------------------- touched cells
// The touched cells listed in the order of the lattice, from the cells' counters: 8 cells per thread,
// one atomic per CTA.  The stencil kernel's own list follows the points; where these are many and lie
// in no order of the lattice (short rods, loose nodes), neighbouring cells are then far apart in the
// list and every kernel of the touched cells fetches the same sectors of the populations again and
// again, from HBM once they exceed the L2 (the rule: ib_list in runtime.cu).  Bound by HBM: 4 B per
// cell (35 us at 4096^2, 8 at 2048^2 inside a step's launches).
__global__ void __launch_bounds__(256) k_ib_list(const RDesc* __restrict__ D, const int* __restrict__ off, int n) {
  __shared__ int s_sum[8], s_base;
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int cells = d.lH * d.lW, c0 = (blockIdx.x - off[r]) * kListCells + threadIdx.x * 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned touched = 0;
  if (c0 + 8 <= cells) {
    const int4 a = *reinterpret_cast<const int4*>(d.ib_cnt + c0), b = *reinterpret_cast<const int4*>(d.ib_cnt + c0 + 4);
    touched = (a.x > 0) | (a.y > 0) << 1 | (a.z > 0) << 2 | (a.w > 0) << 3 | (b.x > 0) << 4 | (b.y > 0) << 5 |
              (b.z > 0) << 6 | (b.w > 0) << 7;
  } else {
    for (int i = 0; i < 8; ++i)
      if (c0 + i < cells && d.ib_cnt[c0 + i] > 0) touched |= 1u << i;
  }
  const int mine = __popc(touched);
  int at = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += v;
  }
  if (lane == 31) s_sum[warp] = at;
  at -= mine;
  __syncthreads();
  int all = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i == warp) at += all;
    all += s_sum[i];
  }
  if (threadIdx.x == 0) s_base = all > 0 ? atomicAdd(d.ib_ctl + 2, all) : 0;
  __syncthreads();
  at += s_base;
  for (; touched; touched &= touched - 1) d.h_new[at++] = c0 + __ffs(touched) - 1;
}

// Sorts R (key, value) pairs in registers by key.
template <int R>
__device__ __forceinline__ void sort_regs(int (&k)[R], float (&w)[R]) {
#pragma unroll
  for (int size = 2; size <= R; size <<= 1)
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int o = i ^ j;
        if (o > i) {
          const bool swap = ((i & size) == 0) ? k[i] > k[o] : k[i] < k[o];
          const int ka = swap ? k[o] : k[i], kb = swap ? k[i] : k[o];
          const float wa = swap ? w[o] : w[i], wb = swap ? w[i] : w[o];
          k[i] = ka;
          k[o] = kb;
          w[i] = wa;
          w[o] = wb;
        }
      }
}

// A head of at most R <= kHeadSort contributions (`first`: the first four of its bucket): its run at
// `start`, its contributions linked to it; returns the coverage (the weights' sum in order of k).
template <int R>
__device__ __forceinline__ float head_row(const RDesc& d, int h, int cell, int len, int4 first, int start, int K2) {
  int k[R];
  float w[R];
  const int4* bucket = reinterpret_cast<const int4*>(d.ib_bucket + (size_t)cell * d.ib_cap);
#pragma unroll
  for (int q = 0; q < R; q += 4) {
    int4 v = first;
    if (q > 0 && q < len) v = bucket[q / 4];
    k[q] = q < len ? v.x : 0x7fffffff;
    k[q + 1] = q + 1 < len ? v.y : 0x7fffffff;
    k[q + 2] = q + 2 < len ? v.z : 0x7fffffff;
    k[q + 3] = q + 3 < len ? v.w : 0x7fffffff;
  }
#pragma unroll
  for (int q = 0; q < R; ++q) w[q] = q < len ? d.ib_w[k[q]] : 0.0f;
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (q < len) d.ib_slot[k[q]] = h;
  sort_regs<R>(k, w);
  float cov = w[0];
#pragma unroll
  for (int q = 1; q < R; ++q)
    if (q < len) cov = cov + w[q];
  int4* row = reinterpret_cast<int4*>(d.run + start);  // runs start at even entries
#pragma unroll
  for (int q = 0; q < R; q += 2)
    if (q < len) {
      const int a = K2 == 16 ? k[q] >> 4 : k[q] / K2, b = K2 == 16 ? k[q + 1] >> 4 : k[q + 1] / K2;
      row[q / 2] = make_int4(a, __float_as_int(w[q]), b, __float_as_int(w[q + 1]));
    }
  return cov;
}

// Sorts n distinct ints by one warp, whose lanes all call it: chunks of 32 in registers, then merges
// of neighbouring runs, every element placed by its rank in the run beside its own.  Element i is at
// a[2 i]; b, as large, is the second buffer.  Returns the one that holds the result.  Bound by the
// merges' dependent loads.  Comparing every pair instead costs n^2 / 32 steps: with 4,096 contributions
// in each of 16 cells, taken by one warp in turn, ordering took 72.9 ms a step; 5.6 now (15.5 with the
// sort by tiles that the buckets replaced).  1,024 in each: 6.8 and 1.2 (3.5); 28 in each of 2,300
// cells: 186 and 172 us (1,067).
__device__ const int* sort_warp(int* a, int* b, int n, int lane) {
  for (int c = 0; c < n; c += 32) {
    int v = c + lane < n ? a[2 * (c + lane)] : 0x7fffffff;
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
      for (int j = size >> 1; j > 0; j >>= 1) {
        const int o = __shfl_xor_sync(0xffffffffu, v, j);
        v = ((lane & j) == 0) == ((lane & size) == 0) ? min(v, o) : max(v, o);
      }
    if (c + lane < n) a[2 * (c + lane)] = v;
  }
  __syncwarp();
  for (int w = 32; w < n; w <<= 1) {
    for (int i = lane; i < n; i += 32) {
      const int first = i / (2 * w) * (2 * w), mid = min(first + w, n), end = min(mid + w, n);
      const int v = a[2 * i];
      int lo = i < mid ? mid : first, hi = i < mid ? end : mid;
      const int other = lo;
      while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (a[2 * m] < v) lo = m + 1; else hi = m;
      }
      b[2 * (first + (lo - other) + (i - (i < mid ? first : mid)))] = v;
    }
    __syncwarp();
    int* const t = a;
    a = b;
    b = t;
  }
  return a;
}

// A head with more contributions than are sorted in registers, by a whole warp: gathered from the bucket
// and the overflow list, sorted, and its run written behind them.
__device__ __forceinline__ float head_pool(const RDesc& d, int h, int cell, int len, int K2, int lane, int& start) {
  int base = 0;
  const int pad = (len + 1) & ~1;
  if (lane == 0) base = atomicAdd(d.ib_ctl + 1, 2 * pad);
  base = __shfl_sync(0xffffffffu, base, 0);
  int2* raw = d.run + base;
  int2* run = raw + pad;
  const int* bucket = d.ib_bucket + (size_t)cell * d.ib_cap;
  const int held = min(len, d.ib_cap);
  for (int i = lane; i < held; i += 32) raw[i].x = bucket[i];
  if (lane == 0 && len > d.ib_cap) {
    int e = d.ib_ovf_head[cell];
    for (int i = d.ib_cap; i < len; ++i) {
      raw[i].x = d.ib_ovf[e];
      e = d.ib_ovf_next[e];
    }
    d.ib_ovf_head[cell] = -1;
  }
  __syncwarp();
  const int* sorted = sort_warp(&raw->x, &raw->y, len, lane);
  for (int i = lane; i < len; i += 32) {
    const int k = sorted[2 * i];
    run[i] = make_int2(k / K2, __float_as_int(d.ib_w[k]));
    d.ib_slot[k] = h;
  }
  __syncwarp();
  float cov = __int_as_float(run[0].y);
  for (int q = 1; q < len; ++q) cov = cov + __int_as_float(run[q].y);
  start = base + pad;
  return cov;
}

// The CTA's heads with more contributions than that (deep), a warp each, shared among its warps: the
// cells around one spot are neighbours in the list.  Returns the coverage (its bits) and the start of
// the calling thread's run.
__device__ __noinline__ int2 deep_heads(const RDesc& d, int h0, int cell, int len, bool deep, int K2) {
  __shared__ int s_deep, s_head[kHeadThreads];
  __shared__ int2 s_cell[kHeadThreads], s_run[kHeadThreads];
  if (threadIdx.x == 0) s_deep = 0;
  s_cell[threadIdx.x] = make_int2(cell, len);
  __syncthreads();
  if (deep) s_head[atomicAdd(&s_deep, 1)] = threadIdx.x;
  __syncthreads();
  for (int i = threadIdx.x >> 5; i < s_deep; i += kHeadThreads / 32) {
    const int t = s_head[i], lane = threadIdx.x & 31;
    int at;
    const float c = head_pool(d, h0 + t, s_cell[t].x, s_cell[t].y, K2, lane, at);
    if (lane == 0) s_run[t] = make_int2(__float_as_int(c), at);
  }
  __syncthreads();
  return s_run[threadIdx.x];
}

// One thread per touched cell: its contributions ordered by k, the coverage -> 1/max(cov, 1), the
// macroscopic state pulled from h[parity] (density, clamped velocity), u_corrected = velocity
// (fluid.py:268-290).  Bound by the latency of its three dependent loads (the cell, its bucket and
// populations, the weights), with every head's loads in flight at once.  A CTA's runs lie one behind
// the other (a scan of their lengths, one atomic per CTA for their place), since every forcing round
// reads them all: per step at 4096^2 with 307,200 points the rounds' spread halves took 349 us with a
// row of 16 entries for each cell and 268 packed (and 1 / coverage apart from the macroscopic
// state), this kernel 154 and 132.
// Before, one CTA per 16x16 tile counting-sorted the tile's contributions in shared memory, in
// phases separated by barriers; a tile with more than 2,048 took a sort in global memory, whose
// tail set the kernel's time on dense rollouts.  Measured (per launch in a step): 1024^2 with
// 16,384 points 26 -> 11.3 us, a batch of 64 uneven rollouts with 74 k points 225 -> 54 us.  Sorting
// up to 8 entries in registers instead of 16 took 46 and 82 us: where rods cross, whole warps of cells
// then took the path of the longer ones.
__global__ void __launch_bounds__(kHeadThreads) k_ib_heads(const RDesc* __restrict__ D, const int* __restrict__ off,
                                                           int n, int parity) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int h0 = (blockIdx.x - off[r]) * blockDim.x;
  const int heads = d.ib_ctl[2];
  if (h0 >= heads) return;
  const int h = h0 + threadIdx.x;
  const bool on = h < heads;
  const int cell = on ? d.h_new[h] : 0;
  const int len = on ? d.ib_cnt[cell] : 0;
  int4 first = make_int4(0, 0, 0, 0);
  if (on) first = *reinterpret_cast<const int4*>(d.ib_bucket + (size_t)cell * d.ib_cap);
  const int lW = d.lW, lH = d.lH, K2 = d.K * d.K;
  const int y = cell / lW, x = cell - y * lW;
  const int xm = x == 0 ? lW - 1 : x - 1, xp = x == lW - 1 ? 0 : x + 1;
  const int HW = lH * lW;
  // populations are pulled from the cell opposite to their direction
  const float* __restrict__ r0 = d.h[parity] + y * lW;
  const float* __restrict__ rm = d.h[parity] + (y == 0 ? lH - 1 : y - 1) * lW;
  const float* __restrict__ rp = d.h[parity] + (y == lH - 1 ? 0 : y + 1) * lW;
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
  const int row = min(kHeadSort, d.ib_cap);  // contributions that are sorted in registers and that a bucket holds
  // places of the runs: a scan over the CTA
  __shared__ int s_sum[kHeadThreads / 32], s_base;
  const int lane = threadIdx.x & 31, pad = len <= row ? (len + 1) & ~1 : 0;
  int start = pad;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, start, o);
    if (lane >= o) start += v;
  }
  if (lane == 31) s_sum[threadIdx.x >> 5] = start;
  start -= pad;
  __syncthreads();
  int all = 0;
#pragma unroll
  for (int i = 0; i < kHeadThreads / 32; ++i) {
    if (i == threadIdx.x >> 5) start += all;
    all += s_sum[i];
  }
  if (threadIdx.x == 0) s_base = atomicAdd(d.ib_ctl + 1, all);
  const bool deep = __syncthreads_or(len > row);
  start += s_base;
  float cov = 0.0f;
  if (len > 0 && len <= 8) cov = head_row<8>(d, h, cell, len, first, start, K2);
  if (len > 8 && len <= row) cov = head_row<kHeadSort>(d, h, cell, len, first, start, K2);
  if (deep) {
    const int2 long_run = deep_heads(d, h0, cell, len, len > row, K2);
    if (len > row) {
      cov = __int_as_float(long_run.x);
      start = long_run.y;
    }
  }
  if (!on) return;
  d.ib_cnt[cell] = 0;
  float rho, vx, vy;
  macroscopic(f, d.vmax, d.vmax_q4, rho, vx, vy);
  d.h_cell[h] = cell;
  d.h_run[h] = make_int2(start, len);
  d.s_mac[h] = make_float4(rho, vx, vy, 0.0f);
  d.s_inv[h] = 1.0f / max_prop(cov, 1.0f);
  d.s_uc[h] = make_float2(vx, vy);
}

// Weighted sum of a head-indexed field over the K*K stencil of one point, in stencil order
// (the reference's sum over axis 1 of values * weights, fluid.py:90-97).  The slots and weights
// are read past the L1: a chained kernel reads them before it waits (after_previous).  FUSED, in a
// kernel that runs all rounds: they are read through the L1, round after round, and the field, which
// other SMs write between the rounds, past it.
template <bool FUSED, typename T>
__device__ __forceinline__ T constant_load(const T* p) {
  return FUSED ? *p : __ldcg(p);
}
template <bool FUSED, typename T>
__device__ __forceinline__ T field_load(const T* p) {
  return FUSED ? __ldcg(p) : *p;
}
template <int K2, bool FUSED = false>
struct Taps {
  int slot[K2];
  float w[K2];
  __device__ __forceinline__ void load(const RDesc& d, int point) {
    const int base = point * K2;
    if (K2 % 4 == 0) {
#pragma unroll
      for (int s = 0; s < K2; s += 4) {
        const int4 q = constant_load<FUSED>(reinterpret_cast<const int4*>(d.ib_slot + base + s));
        const float4 v = constant_load<FUSED>(reinterpret_cast<const float4*>(d.ib_w + base + s));
        slot[s] = q.x; slot[s + 1] = q.y; slot[s + 2] = q.z; slot[s + 3] = q.w;
        w[s] = v.x; w[s + 1] = v.y; w[s + 2] = v.z; w[s + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int s = 0; s < K2; ++s) {
        slot[s] = constant_load<FUSED>(d.ib_slot + base + s);
        w[s] = constant_load<FUSED>(d.ib_w + base + s);
      }
    }
  }
  __device__ __forceinline__ float2 sum(const float2* field) const {
    float2 v[K2];
#pragma unroll
    for (int s = 0; s < K2; ++s) v[s] = field_load<FUSED>(field + slot[s]);
    float x = 0.0f, y = 0.0f;
#pragma unroll
    for (int s = 0; s < K2; ++s) {
      x = x + v[s].x * w[s];
      y = y + v[s].y * w[s];
    }
    return make_float2(x, y);
  }
};
template <int K2, bool FUSED>
__device__ __forceinline__ float2 stencil_sum(const RDesc& d, int point, const float2* field) {
  Taps<K2, FUSED> taps;
  taps.load(d, point);
  return taps.sum(field);
}

template <bool FUSED = false>
__device__ __forceinline__ float2 stencil_sum_any(const RDesc& d, int point, const float2* field) {
  switch (d.K) {
    case 4: return stencil_sum<16, FUSED>(d, point, field);
    case 2: return stencil_sum<4, FUSED>(d, point, field);
    case 3: return stencil_sum<9, FUSED>(d, point, field);
    default: break;
  }
  const int K2 = d.K * d.K;
  float x = 0.0f, y = 0.0f;
  for (int s = 0; s < K2; ++s) {
    const int k = point * K2 + s;
    const float2 v = field_load<FUSED>(field + d.ib_slot[k]);
    const float w = d.ib_w[k];
    x = x + v.x * w;
    y = y + v.y * w;
  }
  return make_float2(x, y);
}

// Body force of a touched cell from its corrected velocity after the last multi-direct
// forcing round (fluid.py:327-339): post clamp of u_corrected, F = (u_c - u) rho, optional
// force clamp.
__device__ __forceinline__ float2 head_force(const RDesc& d, float4 mac, float2 uc) {
  const float c2 = clamp_factor_fast(uc.x, uc.y, d.vmax, d.vmax_q4);
  uc.x = uc.x * c2;
  uc.y = uc.y * c2;
  float Fx = (uc.x - mac.y) * mac.x;
  float Fy = (uc.y - mac.z) * mac.x;
  if (d.force_clamp) {
    const float c3 = clamp_factor(Fx, Fy, d.vmax);
    Fx = Fx * c3;
    Fy = Fy * c3;
  }
  return make_float2(Fx, Fy);
}

// The correction of one point from u at the point (fluid.py:297-302).
__device__ __forceinline__ void ib_correct(const RDesc& d, int p, float2 v, float2 u) {
  const float sx = (v.x - u.x) * d.relax;
  const float sy = (v.y - u.y) * d.relax;
  const float cf = clamp_factor_fast(sx, sy, d.vmax, d.vmax_q4);
  d.delta[p] = make_float2(sx * cf, sy * cf);
}

// What a round reads that its predecessor does not write is read before the wait: after the first
// round the predecessor is k_ib_spread, which writes s_uc and s_f, and the point's velocity, slots
// and weights are older.
template <int K2>
__device__ __forceinline__ void interp_point(const RDesc& d, int p, bool on, int it) {
  if (it == 0) after_previous();  // k_ib_heads writes the slots
  Taps<K2> taps;
  float2 v;
  if (on) {
    v = __ldcg(d.nvl + p);
    taps.load(d, p);
  }
  if (it > 0) after_previous();
  if (on) ib_correct(d, p, v, taps.sum(d.s_uc));
}

// Multi-direct forcing, interpolation half (fluid.py:292-302): per IB point, u at the point
// = sum_s w_s u_corrected(cell_s); correction = (U_point - u) * relaxation, clamped.
__global__ void __launch_bounds__(256) k_ib_interp(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                   int it) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const int p = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;  // IB point
  const bool on = p < d.NI && it < d.ib_iters;
  switch (d.K) {
    case 4: return interp_point<16>(d, p, on, it);
    case 2: return interp_point<4>(d, p, on, it);
    case 3: return interp_point<9>(d, p, on, it);
    default: break;
  }
  after_previous();
  if (on) ib_correct(d, p, d.nvl[p], stencil_sum_any(d, p, d.s_uc));
}

// In-order sum of correction * weight over a head's run (fluid.py:304-309).  Runs are short: 8
// entries are fetched at a time (those that exist) so that all their loads are in flight together.
template <bool FUSED = false>
struct RunChunk {
  int4 e[4];
  __device__ __forceinline__ void load(const int2* run, int len, int j) {
    const int4* pairs = reinterpret_cast<const int4*>(run);  // runs start at even entries
#pragma unroll
    for (int q = 0; q < 4; ++q)
      e[q] = j + 2 * q < len ? constant_load<FUSED>(pairs + j / 2 + q) : make_int4(0, 0, 0, 0);
  }
  __device__ __forceinline__ void add(int len, int j, const float2* delta, float2& sum) const {
    float2 v[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[2 * q] = j + 2 * q < len ? field_load<FUSED>(delta + e[q].x) : make_float2(0.0f, 0.0f);
      v[2 * q + 1] = j + 2 * q + 1 < len ? field_load<FUSED>(delta + e[q].z) : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (j + 2 * q < len) {
        sum.x = sum.x + v[2 * q].x * __int_as_float(e[q].y);
        sum.y = sum.y + v[2 * q].y * __int_as_float(e[q].y);
      }
      if (j + 2 * q + 1 < len) {
        sum.x = sum.x + v[2 * q + 1].x * __int_as_float(e[q].w);
        sum.y = sum.y + v[2 * q + 1].y * __int_as_float(e[q].w);
      }
    }
  }
};

// Multi-direct forcing, spread half (fluid.py:304-310): per touched cell, the in-order sum
// of correction * weight over its contributions, times 1/max(coverage, 1), added to
// u_corrected.
__global__ void __launch_bounds__(256) k_ib_spread(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                   int it, int fuse_finalize) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const int p = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  // the plan's last round also computes each touched cell's body force (k_ib_finalize's
  // work for the same cell) when every rollout of the plan runs the same number of rounds
  const bool fin = fuse_finalize && it == d.ib_iters - 1;
  // the predecessor, k_ib_interp, writes delta only: all else is read before the wait for it
  const int heads = __ldcg(d.ib_ctl + 2);
  const bool on = it < d.ib_iters && p < heads;
  int2 run = make_int2(0, 0);
  float4 mac;
  float2 u;
  float inv;
  if (on) {
    run = __ldcg(d.h_run + p);
    inv = __ldcg(d.s_inv + p);
    u = __ldcg(d.s_uc + p);
    if (fin) mac = __ldcg(d.s_mac + p);
  }
  RunChunk<> c;
  c.load(d.run + run.x, run.y, 0);
  after_previous();
  if (fin && p == 0) d.ib_ctl[5] = heads;
  if (!on) return;
  float2 s = make_float2(0.0f, 0.0f);
  c.add(run.y, 0, d.delta, s);
  for (int j = 8; j < run.y; j += 8) {
    c.load(d.run + run.x, run.y, j);
    c.add(run.y, j, d.delta, s);
  }
  u = make_float2(u.x + s.x * inv, u.y + s.y * inv);
  d.s_uc[p] = u;
  if (fin) d.s_f[p] = head_force(d, mac, u);
}

// ---------------------------------------------------------------- fused IB iterations
// Barrier among the CTAs of one rollout inside a cooperative launch (all CTAs resident).
// The spin is bounded: on timeout the rollout's MC_FLAG_TIMEOUT is set and the kernel
// continues (its results are then invalid) instead of hanging the device.
__device__ __forceinline__ void rollout_barrier(int* ctl, int nb, unsigned* flags) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile int* gen = ctl + 4;
    const int g = *gen;
    __threadfence();
    if (atomicAdd(ctl + 3, 1) == nb - 1) {
      atomicExch(ctl + 3, 0);
      __threadfence();
      atomicAdd(ctl + 4, 1);
    } else {
      unsigned it = 0;
      while (*gen == g) {
        if (++it > (1u << 22)) {
          atomicOr(flags, 2u);
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// All ibm_iterations of the multi-direct forcing and the body force of every rollout in one
// cooperative launch: [interpolate (nodes) | barrier | spread (touched cells) | barrier] x
// iterations, then the finalize of every touched cell.  Same arithmetic and order as
// k_ib_interp / k_ib_spread / k_ib_finalize, and the same loads of whole vectors (with loads of single
// slots, weights and entries instead: 1024^2 162 us a step, in clusters of 8 CTAs 352; 139 and 213 so);
// values written in one phase and read in the next are loaded past the SM's L1.
// The shared body: threads t0, t0 + stride, ... of one rollout; `sync` is the barrier among
// all of the rollout's threads.
template <typename Sync>
__device__ __forceinline__ void ib_iterations(const RDesc& d, int t0, int stride, Sync sync) {
  const int nheads = __ldcg(d.ib_ctl + 2);
  for (int it = 0; it < d.ib_iters; ++it) {
    for (int p = t0; p < d.NI; p += stride) {  // IB points
      const float2 u = stencil_sum_any<true>(d, p, d.s_uc);
      const float2 nv = d.nvl[p];
      const float sx = (nv.x - u.x) * d.relax;
      const float sy = (nv.y - u.y) * d.relax;
      const float cf = clamp_factor(sx, sy, d.vmax);
      d.delta[p] = make_float2(sx * cf, sy * cf);
    }
    sync();
    for (int p = t0; p < nheads; p += stride) {
      const int2 run = d.h_run[p];
      float2 s = make_float2(0.0f, 0.0f);
      RunChunk<true> c;
      for (int j = 0; j < run.y; j += 8) {
        c.load(d.run + run.x, run.y, j);
        c.add(run.y, j, d.delta, s);
      }
      const float inv = d.s_inv[p];
      const float2 u = __ldcg(d.s_uc + p);
      d.s_uc[p] = make_float2(u.x + s.x * inv, u.y + s.y * inv);
    }
    sync();
  }
  for (int p = t0; p < nheads; p += stride) d.s_f[p] = head_force(d, d.s_mac[p], __ldcg(d.s_uc + p));
  if (t0 == 0) d.ib_ctl[5] = nheads;  // for k_collide_heads
}

__global__ void __launch_bounds__(256) k_ib_coop(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                 int parity) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  const int nb = off[r + 1] - off[r];
  const int lb = blockIdx.x - off[r];
  ib_iterations(d, lb * blockDim.x + threadIdx.x, nb * blockDim.x,
                [&] { rollout_barrier(d.ib_ctl, nb, d.flags); });
}

// The same iterations with one thread-block cluster per rollout (cluster c = rollout c):
// the hardware cluster barrier (release / acquire at cluster scope) separates the phases,
// so a rollout's 2 x iterations + 1 dependent steps cost no kernel boundaries and no
// software barrier.  Every CTA of a cluster reaches every barrier: the early return below
// is uniform across the cluster.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int T>
__global__ void __launch_bounds__(T) k_ib_cluster(const RDesc* __restrict__ D, int n) {
  unsigned rank, ncta, cid;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
  asm("mov.u32 %0, %%clusterid.x;" : "=r"(cid));
  if ((int)cid >= n) return;
  const RDesc& d = D[cid];
  if (!d.enable_fluid || d.NI == 0) return;
  ib_iterations(d, (int)(rank * blockDim.x + threadIdx.x), (int)(ncta * blockDim.x), [] { cluster_sync_all(); });
}

// Post-accumulation clamp and body force F = (u_corrected - u) rho (fluid.py:327-339) per
// touched cell, for the node reaction and for k_collide_heads, which collides these cells
// after the dense pass.  The head count is saved in ib_ctl[5] for k_collide_heads.
__global__ void __launch_bounds__(256) k_ib_finalize(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                     int parity) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int p = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  const int nheads = d.ib_ctl[2];
  if (p == 0) d.ib_ctl[5] = nheads;
  if (p >= nheads) return;
  d.s_f[p] = head_force(d, d.s_mac[p], d.s_uc[p]);
}

// Node reaction (fluid.py:364-382), final wrap (simulate.py:97-98), non-finite check and
// per-step node recording (simulate.py:21-32).
__global__ void __launch_bounds__(256) k_reaction(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                                  const int* tdev) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  after_previous();
  const int node = (blockIdx.x - off[r]) * blockDim.x + threadIdx.x;
  if (node == 0) {
    // this step's deposit has been reduced: reset the CIC bin controls
    d.c_ctl[0] = 0;
    d.c_ctl[1] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d.wl_ctl[1] = 0;  // the plan's CIC tile list and its cursor
    d.wl_ctl[3] = 0;
  }
  if (node >= d.N) return;
  float vx = d.vel[2 * node], vy = d.vel[2 * node + 1];
  if (d.enable_fluid) {
    float2 f = stencil_sum_any(d, node, d.s_f);
    if (d.NI > d.N) {
      // synthetic pair: the mean of the two points' forces (fluid.py:371-374)
      const float2 g = stencil_sum_any(d, node + d.N, d.s_f);
      f = make_float2(0.5f * (f.x + g.x), 0.5f * (f.y + g.y));
    }
    vx = vx - (f.x / d.node_mass) / d.sdt_x;
    vy = vy - (f.y / d.node_mass) / d.sdt_y;
    d.vel[2 * node] = vx;
    d.vel[2 * node + 1] = vy;
  }
  const float px = fmod_floor(d.pos[2 * node], (float)d.W);
  const float py = fmod_floor(d.pos[2 * node + 1], (float)d.H);
  d.pos[2 * node] = px;
  d.pos[2 * node + 1] = py;
  if (!(isfinite(px) && isfinite(py) && isfinite(vx) && isfinite(vy))) atomicOr(d.flags, 1u);
  if (d.rec_every > 0) {
    const int t = *tdev;
    if ((t + 1) % d.rec_every == 0) {
      const size_t e = (size_t)((t + 1) / d.rec_every - 1) * d.N * 2;
      if (d.rec_pos) {
        d.rec_pos[e + 2 * node] = px;
        d.rec_pos[e + 2 * node + 1] = py;
      }
      if (d.rec_vel) {
        d.rec_vel[e + 2 * node] = vx;
        d.rec_vel[e + 2 * node + 1] = vy;
      }
    }
  }
}

// One output sample of a linear, antialiased resize along one axis (JAX's image resize,
// method "linear": triangle kernel widened by max(m/n, 1), weights normalised by their sum
// over the input, zero outside the sampled range): input m -> output n, output index o.
// Writes the first input index and up to kResizeTaps normalised weights; returns the count.
constexpr int kResizeTaps = 16;
__device__ int resize_taps(int o, int m, int n, float inv, float ks, int& i0, float* w) {
  if (m == n) {
    i0 = o;
    w[0] = 1.0f;
    return 1;
  }
  const float sf = ((float)o + 0.5f) * inv - 0.5f;
  int a = (int)floorf(sf - ks), b = (int)ceilf(sf + ks);
  a = a < 0 ? 0 : a;
  b = b > m - 1 ? m - 1 : b;
  if (b - a + 1 > kResizeTaps) b = a + kResizeTaps - 1;  // plans keep the support within the taps
  float tot = 0.0f;
  for (int i = a; i <= b; ++i) {
    float x = fabsf(sf - (float)i) / ks;
    const float v = 1.0f - fabsf(x);
    w[i - a] = v > 0.0f ? v : 0.0f;
    tot = tot + w[i - a];
  }
  const bool inside = sf >= -0.5f && sf <= (float)m - 0.5f;
  const bool norm = fabsf(tot) > 1000.0f * MC_EPSIL;
  for (int i = a; i <= b; ++i) w[i - a] = (inside && norm) ? w[i - a] / tot : 0.0f;
  i0 = a;
  return b - a + 1;
}

// Per-step field recording (steric, fluid_velocity) on recording steps.  The recorded u*
// is on the domain grid: a copy when the lattice is the domain grid, else the linear
// resize of simulate.py:24-29.
__global__ void k_record_fields(const RDesc* __restrict__ D, const int* __restrict__ off, int n,
                                const int* __restrict__ tdev, int advanced) {
  const int r = find_rollout(off, n, blockIdx.x);
  const RDesc& d = D[r];
  if (d.rec_every <= 0) return;
  const int t = *tdev - advanced;  // advanced: the step counter already stands at the next step
  if ((t + 1) % d.rec_every != 0) return;
  const size_t e = (size_t)((t + 1) / d.rec_every - 1);
  const size_t HW = (size_t)d.H * d.W, LHW = (size_t)d.lH * d.lW;
  const bool same = d.lH == d.H && d.lW == d.W;
  const size_t stride = (size_t)(off[r + 1] - off[r]) * blockDim.x;
  for (size_t i = (size_t)(blockIdx.x - off[r]) * blockDim.x + threadIdx.x; i < HW; i += stride) {
    if (d.rec_steric) d.rec_steric[e * HW + i] = d.steric[i];
    if (!d.rec_fluid) continue;
    if (same) {
      d.rec_fluid[e * 2 * HW + i] = d.fluid_vel[i];
      d.rec_fluid[e * 2 * HW + HW + i] = d.fluid_vel[HW + i];
      continue;
    }
    const int y = (int)(i / d.W), x = (int)(i - (size_t)y * d.W);
    float wy[kResizeTaps], wx[kResizeTaps];
    int y0, x0;
    const int ny = resize_taps(y, d.lH, d.H, d.rs_inv_y, d.rs_ks_y, y0, wy);
    const int nx = resize_taps(x, d.lW, d.W, d.rs_inv_x, d.rs_ks_x, x0, wx);
    for (int c = 0; c < 2; ++c) {
      const float* u = d.fluid_vel + c * LHW;
      float acc = 0.0f;
      for (int a = 0; a < ny; ++a) {
        float row = 0.0f;
        for (int b = 0; b < nx; ++b) row = row + wx[b] * u[(size_t)(y0 + a) * d.lW + x0 + b];
        acc = acc + wy[a] * row;
      }
      d.rec_fluid[e * 2 * HW + c * HW + i] = acc;
    }
  }
}

__global__ void k_tick(int* tdev) {
  after_previous();
  *tdev += 1;
}

cudaError_t tiles_blocks_per_sm(int threads, int capS, int* out) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k_bin_tiles, threads, (size_t)4 * capS * sizeof(unsigned));
}
void launch_bin_tiles(const Launch& L, const int2* wl, int* wl_count, int capS, int threads) {
  launch(L, k_bin_tiles, threads, (size_t)4 * capS * sizeof(unsigned), L.d, wl, wl_count, capS);
}
void launch_ib_list(const Launch& L) { launch(L, k_ib_list, kListCells / 8, 0, L.d, L.off, L.n); }
void launch_ib_heads(const Launch& L, int parity) {
  launch(L, k_ib_heads, kHeadThreads, 0, L.d, L.off, L.n, parity);
}
// `bytes` is the per-block opt-in limit; the kernel's static shared memory comes off it.
cudaError_t tiles_set_smem(size_t bytes) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_bin_tiles);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_bin_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(bytes - a.sharedSizeBytes));
}
void launch_ib_interp(const Launch& L, int it) { launch(L, k_ib_interp, kNodeThreads, 0, L.d, L.off, L.n, it); }
void launch_ib_spread(const Launch& L, int it, int fuse_finalize) {
  launch(L, k_ib_spread, kHeadThreads, 0, L.d, L.off, L.n, it, fuse_finalize);
}
cudaError_t launch_ib_coop(const Launch& L, int parity) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L.grid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = L.s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_ib_coop, L.d, L.off, L.n, parity);
}
// One cluster of `ctas` CTAs of `threads` (256 or 1024) threads per rollout (1 <= ctas <=
// 16; above 8 the non-portable size is allowed on the kernel first).
cudaError_t launch_ib_cluster(const RDesc* d, int n, int ctas, int threads, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n * ctas));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (threads == 1024) return cudaLaunchKernelEx(&cfg, k_ib_cluster<1024>, d, n);
  return cudaLaunchKernelEx(&cfg, k_ib_cluster<256>, d, n);
}
cudaError_t ib_cluster_allow_16() {
  cudaError_t e = cudaFuncSetAttribute(k_ib_cluster<256>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_ib_cluster<1024>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
cudaError_t ib_coop_blocks_per_sm(int* out) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k_ib_coop, 256, 0);
}

void launch_ib_finalize(const Launch& L, int parity) {
  launch(L, k_ib_finalize, kHeadThreads, 0, L.d, L.off, L.n, parity);
}
void launch_reaction(const Launch& L, const int* tdev) {
  launch(L, k_reaction, kNodeThreads, 0, L.d, L.off, L.n, tdev);
}
void launch_record_fields(const Launch& L, const int* tdev, int advanced) {
  k_record_fields<<<L.grid, 256, 0, L.s>>>(L.d, L.off, L.n, tdev, advanced);
}
void launch_tick(const Launch& L, int* tdev) {
  Launch one = L;
  one.grid = 1;
  launch(one, k_tick, 1, 0, tdev);
}

}  // namespace mc
