// Comparisons of the rods' branch-free arithmetic (csrc/rod.cuh) with the plain operations it stands
// for; compiled and called by test_gpu_rod_arithmetic.py.  Every entry returns a CUDA error code and
// counts, in `bad` (device, zeroed by the caller), the operands for which the results differ.
#include "../microcosmos_b200/csrc/rod.cuh"

using namespace mc;

namespace {

using u64 = unsigned long long;

__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
// a quotient of zero may lose its sign
__device__ bool differ_but_zero(float a, float b) { return differ(a, b) && !(a == 0.0f && b == 0.0f); }

struct Random {
  u64 x;
  __device__ Random(u64 seed, u64 i) : x((seed + i) * 0x9E3779B97F4A7C15ull + 0x2545F4914F6CDD1Dull) {
    for (int k = 0; k < 4; ++k) next();
  }
  __device__ u64 next() {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return x;
  }
  __device__ float uniform() { return (float)(next() >> 40) * 0x1p-24f; }
  // any significand; half of them near a power of two or with few bits
  __device__ unsigned significand() {
    const u64 r = next();
    const unsigned m = (unsigned)r & 0x7fffffu, kind = (unsigned)(r >> 60);
    if (kind < 8) return m;
    if (kind < 10) return m & 3u;
    if (kind < 12) return 0x7fffffu - (m & 3u);
    if (kind < 14) return m & 0x7c0000u;
    return (1u << (m % 23)) | (m >> 20);
  }
  // exponents lo..hi
  __device__ float value(int lo, int hi) {
    return __uint_as_float(((unsigned)(127 + lo + (int)(next() % (u64)(hi - lo + 1))) << 23) | significand());
  }
  __device__ float signed_value(int lo, int hi) {
    const float v = value(lo, hi);
    return next() >> 63 ? -v : v;
  }
};

// every significand of [1, 4) times 2^e, e even from lo to hi: the length of a segment of that
// squared length (its direction is not looked at)
__global__ void k_root(int lo, int hi, u64* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const float s = __uint_as_float(0x3f800000u + i);
  for (int e = lo; e <= hi; e += 2) {
    const float t = ldexpf(s, e);
    float L;
    unit_near(make_float2(1.0f, 1.0f), t, L);
    if (differ(L, sqrtf(t))) atomicAdd(bad, 1ull);
  }
}

// every significand times 2^e, e from lo to hi
__global__ void k_reciprocal(int lo, int hi, u64* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  for (int e = lo; e <= hi; ++e) {
    const float b = ldexpf(__uint_as_float(0x3f800000u + i), e);
    if (differ(reciprocal(b), 1.0f / b)) atomicAdd(bad, 1ull);
  }
}

// quotients over the stated range: a zero or 2^-80 to 2^80, b 2^-30 to 2^30, both ends included
__global__ void k_quotient(u64 seed, int count, u64* bad) {
  Random g(seed, blockIdx.x * blockDim.x + threadIdx.x);
  for (int k = 0; k < count; ++k) {
    float a = g.signed_value(-80, 79), b = g.value(-30, 29);
    const unsigned kind = (unsigned)(g.next() >> 59);
    if (kind == 0) a = copysignf(0x1p-80f, a);
    if (kind == 1) a = copysignf(0x1p80f, a);
    if (kind == 2) b = 0x1p-30f;
    if (kind == 3) b = 0x1p30f;
    if (kind == 4) a = 0.0f;
    if (differ_but_zero(div_near(a, b, reciprocal(b)), a / b)) atomicAdd(bad, 1ull);
  }
}

// direction and length of segments: components that are multiples of 2^-23, as differences by the
// nearest image are, of every size up to 2^17; also axis-parallel and nearly so
__global__ void k_unit(u64 seed, int count, u64* bad) {
  Random g(seed, blockIdx.x * blockDim.x + threadIdx.x);
  for (int k = 0; k < count; ++k) {
    float2 v = make_float2(g.signed_value(-23, 16), g.signed_value(-23, 16));
    if ((g.next() & 3) == 0) v.y = ldexpf(v.x, (int)(g.next() % 3) - 1);
    if ((g.next() & 15) == 0) v.y = 0.0f;
    v.x = rintf(v.x * 0x1p23f) * 0x1p-23f;
    v.y = rintf(v.y * 0x1p23f) * 0x1p-23f;
    const float s = v.x * v.x + v.y * v.y;
    if (!(s >= kNearLength2)) continue;
    float L;
    const float2 u = unit_near(v, s, L);
    const float R = sqrtf(s), Rc = max_prop(R, 1e-8f);
    if (differ(L, R) || differ_but_zero(u.x, v.x / Rc) || differ_but_zero(u.y, v.y / Rc)) atomicAdd(bad, 1ull);
  }
}

// one-period modulo over its range |d| < 1.49 y
__global__ void k_modulo(u64 seed, int count, u64* bad) {
  Random g(seed, blockIdx.x * blockDim.x + threadIdx.x);
  for (int k = 0; k < count; ++k) {
    const float y = (g.next() & 1) ? MC_2PI_F : (float)(4 + g.next() % 16381);
    float d = (2.0f * g.uniform() - 1.0f) * (kNear * y);
    const unsigned kind = (unsigned)(g.next() >> 60);
    if (kind < 4) d = (kind & 1 ? y : -y) * 0.5f + g.signed_value(-40, -5);
    if (kind == 4) d = g.signed_value(-60, 0);
    if (!(fabsf(d) < kNear * y)) continue;
    const float x = d + y / 2.0f;
    if (differ_but_zero(fmod_near(x, y), fmod_floor(x, y))) atomicAdd(bad, 1ull);
  }
}

// One rod of at most 32 nodes per CTA of one warp, its iterations on both paths.  The fast path
// reports (out_left) whether some operand left its range; where none did, the results have to be the
// same bits.  kind 0: ordinary rods; 1: two nodes on one spot; 2: an angle far off; 3: a node
// ten domains away.
__global__ void __launch_bounds__(32) k_rod(u64 seed, int solver, int cycles, int kind, u64* bad, int* out_left) {
  __shared__ float2 tab[chain_smem(32)];
  __shared__ RDesc d;
  const int lane = threadIdx.x;
  Random common(seed, blockIdx.x), g(seed + 77, (u64)blockIdx.x * 32 + lane);
  const int nn = 2 + (int)(common.next() % 31);
  const float scale = exp2f(16.0f * common.uniform() - 11.0f);  // segments of 2^-11 to 2^5
  const int W = 8 + (int)(common.next() % 2000), H = 8 + (int)(common.next() % 2000);
  const float shear = common.uniform(), stretch = common.uniform(), inertia = common.uniform();
  if (lane == 0) {
    d.W = W;
    d.H = H;
    d.cycles = cycles;
    d.k_shear = shear;
    d.k_stretch = solver ? exp2f(14.0f * stretch) : stretch;
    d.cos_w = exp2f(8.0f + 8.0f * inertia);
  }
  __syncwarp();
  const float Wf = (float)d.W, Hf = (float)d.H;
  RodLane l;
  l.j = lane;
  l.nn = nn;
  l.ne = nn - 1;
  l.nb = nn > 2 ? nn - 2 : 0;
  l.own = lane < nn;
  const Team tm = {0, 1, 1};
  const float l0 = scale * (0.5f + g.uniform()), ra = g.uniform() - 0.5f, kb = g.uniform();
  const float dir = 6.2831853f * common.uniform();
  float th = dir + 0.5f * (g.uniform() - 0.5f);
  float x = Wf * common.uniform() + lane * scale * cosf(dir) + 0.2f * scale * g.uniform();
  float y = Hf * common.uniform() + lane * scale * sinf(dir) + 0.2f * scale * g.uniform();
  x = fmod_floor(x, Wf);
  y = fmod_floor(y, Hf);
  const int odd = nn / 2 - 1;
  const float xo = __shfl_sync(0xffffffffu, x, odd), yo = __shfl_sync(0xffffffffu, y, odd);
  if (kind == 1 && lane == odd + 1) x = xo, y = yo;
  if (kind == 2 && lane == odd) th += 40.0f;
  if (kind == 3 && lane == odd) x += 10.6f * Wf;
  const float edg = ((lane < l.nb) + (lane >= 1 && lane - 1 < l.nb)) == 2 ? 0.5f : 1.0f;
  const float ndg = ((lane < l.ne) + (lane >= 1 && lane - 1 < l.ne)) == 2 ? 0.5f : 1.0f;
  float rx[2], ry[2], rt[2];
  bool left = false;
  for (int near = 1; near >= 0; --near) {
    float px = x, py = y, t = th;
    bool out;
    if (solver == 1) {
      float2* ex = tab + kThetaChunk * 32;
      float* ext = reinterpret_cast<float*>(tab);
      out = near ? cosserat_iterations<true, false>(d, tm, l, px, py, t, l0, ra, kb, edg, ex, ext, 32)
                 : cosserat_iterations<false, false>(d, tm, l, px, py, t, l0, ra, kb, edg, ex, ext, 32);
    } else {
      // one chunk: the angles, the rest vectors, the positions
      out = near ? theta_passes<true, false>(tm, l, cycles, t, ra, kb, edg, tab, 32)
                 : theta_passes<false, false>(tm, l, cycles, t, ra, kb, edg, tab, 32);
      __syncwarp();
      for (int k = 0; k < cycles && lane < l.ne; ++k) {
        float sn, cs;
        sincosf(tab[k * 32 + lane].x, &sn, &cs);
        tab[k * 32 + lane] = make_float2(cs * l0, sn * l0);
      }
      __syncwarp();
      int buf = 0;
      const bool o2 =
          near ? position_passes<true, false>(tm, l, cycles, true, px, py, l0, ndg, Wf, Hf, d.k_shear, d.k_stretch, tab,
                                              tab, buf, 32)
               : position_passes<false, false>(tm, l, cycles, true, px, py, l0, ndg, Wf, Hf, d.k_shear, d.k_stretch,
                                               tab, tab, buf, 32);
      out = out || o2;
      __syncwarp();
    }
    if (near) left = __any_sync(0xffffffffu, out);
    rx[near] = px;
    ry[near] = py;
    rt[near] = t;
  }
  const bool same = !(lane < nn) || (!differ(rx[0], rx[1]) && !differ(ry[0], ry[1]) && (lane >= l.ne || !differ(rt[0], rt[1])));
  if (lane == 0 && left) atomicAdd(out_left, 1);
  if (!left && !__all_sync(0xffffffffu, same) && lane == 0) atomicAdd(bad, 1ull);
}

}  // namespace

extern "C" {
int check_root(int lo, int hi, u64* bad) {
  k_root<<<(1 << 24) / 256, 256>>>(lo, hi, bad);
  return cudaDeviceSynchronize();
}
int check_reciprocal(int lo, int hi, u64* bad) {
  k_reciprocal<<<(1 << 23) / 256, 256>>>(lo, hi, bad);
  return cudaDeviceSynchronize();
}
int check_quotient(u64 seed, u64* bad) {
  k_quotient<<<1024, 256>>>(seed, 2000, bad);
  return cudaDeviceSynchronize();
}
int check_unit(u64 seed, u64* bad) {
  k_unit<<<1024, 256>>>(seed, 2000, bad);
  return cudaDeviceSynchronize();
}
int check_modulo(u64 seed, u64* bad) {
  k_modulo<<<1024, 256>>>(seed, 2000, bad);
  return cudaDeviceSynchronize();
}
int check_rods(int rods, u64 seed, int solver, int cycles, int kind, u64* bad, int* out_left) {
  if (cycles < 1 || cycles > kThetaChunk) return cudaErrorInvalidValue;
  k_rod<<<rods, 32>>>(seed, solver, cycles, kind, bad, out_left);
  return cudaDeviceSynchronize();
}
}
