// k_pme.cu -- reciprocal-space PME: B-spline spread, 3D real-to-complex FFT
// with the Ewald convolution fused into the x pass, complex-to-real FFT, and
// the force gather.
//
// Physics follows src/gpu/kernels/pme.wgsl:124 (spread), fft.wgsl:60,
// pme-convolve.wgsl:34, pme-interpolate.wgsl:105 and the f64 oracle
// src/reference/forces/pme.ts:93-263: order-5 cardinal B-splines on a mesh
// laid out in fractional coordinates, E = sum_k f(k) |Q(k)|^2 with
// f = (2 pi / V) ONE_4PI_EPS0 exp(-k^2/4a^2) / (k^2 |b(m)|^2), and the grid
// multiplied by 2 f before the inverse transform.
//
// B200 shape:
//   * the spline argument u = r . (K o B^-1) is formed exactly in 2^32 fixed
//     point from the int64 positions (a 64x64->128-bit product), so the grid
//     index and the weight fraction carry no f32 coordinate rounding;
//   * the charge grid is int64 fixed point filled with atomics, so the spread
//     is order independent and runs are bit-identical;
//   * the transform is three passes, each CTA running a Stockham mixed-radix
//     (2 to 10) FFT over whole lines in shared memory: one CTA per
//     x-plane does z (int64 -> complex, real-to-complex, clearing the grid it
//     read) and y; the x pass does x forward + convolution + x inverse; one
//     CTA per x-plane does y inverse and z complex-to-real.  Meshes whose
//     planes do not fit shared memory take separate z and y passes (five in
//     all).  The reference's 7-13 global passes per direction and its
//     separate load/convolve passes disappear.
#include <array>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "device_state.h"
#include "prep.h"

namespace mdb {
namespace {

constexpr int kThreads = 256;

// ------------------------------------------------------------ transforms --
// Discrete transforms of R values in registers, R = 2 .. 10, so that most mesh
// axes of up to 100 points take two passes through shared memory (75, 84, 96
// and 98 take three).  SIGN is
// the exponent's (-1 forward, +1 inverse).  Products that feed a sum are
// written as fused steps, so every kernel that runs a line gives the same bits.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
template <int SIGN>
__device__ __forceinline__ float2 times_i(float2 a) {
  return SIGN < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}
// a + c b and a + SIGN i c b
__device__ __forceinline__ float2 axpy(float c, float2 b, float2 a) { return make_float2(fmaf(c, b.x, a.x), fmaf(c, b.y, a.y)); }

template <int SIGN>
__device__ __forceinline__ void dft2(float2& a, float2& b) {
  const float2 s = cadd(a, b);
  b = csub(a, b);
  a = s;
}
template <int SIGN>
__device__ __forceinline__ void dft3(float2& a, float2& b, float2& c) {
  const float2 t = cadd(b, c), u = axpy(-0.5f, t, a);
  const float2 w = times_i<SIGN>(make_float2(__fmul_rn(0.866025404f, b.x - c.x), __fmul_rn(0.866025404f, b.y - c.y)));
  a = cadd(a, t);
  b = cadd(u, w);
  c = csub(u, w);
}
template <int SIGN>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
  const float2 p = cadd(a, c), q = csub(a, c), r = cadd(b, d), s = times_i<SIGN>(csub(b, d));
  a = cadd(p, r);
  c = csub(p, r);
  b = cadd(q, s);
  d = csub(q, s);
}
template <int SIGN>
__device__ __forceinline__ void dft5(float2& a, float2& b, float2& c, float2& d, float2& e) {
  const float c1 = 0.309016994f, c2 = -0.809016994f, s1 = 0.951056516f, s2 = 0.587785252f;
  const float2 t1 = cadd(b, e), t2 = cadd(c, d), t3 = csub(b, e), t4 = csub(c, d);
  const float2 m1 = axpy(c2, t2, axpy(c1, t1, a)), m2 = axpy(c1, t2, axpy(c2, t1, a));
  const float2 n1 = times_i<SIGN>(axpy(s2, t4, make_float2(__fmul_rn(s1, t3.x), __fmul_rn(s1, t3.y))));
  const float2 n2 = times_i<SIGN>(axpy(-s1, t4, make_float2(__fmul_rn(s2, t3.x), __fmul_rn(s2, t3.y))));
  a = cadd(a, cadd(t1, t2));
  b = cadd(m1, n1);
  e = csub(m1, n1);
  c = cadd(m2, n2);
  d = csub(m2, n2);
}

template <int R, int SIGN>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 2) dft2<SIGN>(v[0], v[1]);
  else if constexpr (R == 3) dft3<SIGN>(v[0], v[1], v[2]);
  else if constexpr (R == 4) dft4<SIGN>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 5) dft5<SIGN>(v[0], v[1], v[2], v[3], v[4]);
  else if constexpr (R == 7) {
    const float c1 = 0.623489802f, c2 = -0.222520934f, c3 = -0.900968868f;
    const float s1 = 0.781831482f, s2 = 0.974927912f, s3 = 0.433883739f;
    const float2 p1 = cadd(v[1], v[6]), p2 = cadd(v[2], v[5]), p3 = cadd(v[3], v[4]);
    const float2 q1 = csub(v[1], v[6]), q2 = csub(v[2], v[5]), q3 = csub(v[3], v[4]);
    auto even = [&](float a, float b, float c) { return axpy(c, p3, axpy(b, p2, axpy(a, p1, v[0]))); };
    auto odd = [&](float a, float b, float c) {
      return times_i<SIGN>(axpy(c, q3, axpy(b, q2, make_float2(__fmul_rn(a, q1.x), __fmul_rn(a, q1.y)))));
    };
    const float2 e1 = even(c1, c2, c3), e2 = even(c2, c3, c1), e3 = even(c3, c1, c2);
    const float2 o1 = odd(s1, s2, s3), o2 = odd(s2, -s3, -s1), o3 = odd(s3, -s1, s2);
    v[0] = cadd(v[0], cadd(p1, cadd(p2, p3)));
    v[1] = cadd(e1, o1);
    v[6] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[5] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[4] = csub(e3, o3);
  } else if constexpr (R == 8) {
    dft4<SIGN>(v[0], v[2], v[4], v[6]);
    dft4<SIGN>(v[1], v[3], v[5], v[7]);
    const float h = 0.707106781f;
    const float2 w1 = make_float2(h, SIGN * h), w3 = make_float2(-h, SIGN * h);
    const float2 o1 = cmul(v[3], w1), o2 = times_i<SIGN>(v[5]), o3 = cmul(v[7], w3);
    const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  } else if constexpr (R == 9) {
#pragma unroll
    for (int n = 0; n < 3; ++n) dft3<SIGN>(v[n], v[n + 3], v[n + 6]);  // v[n + 3 k] holds component k of column n
    const float2 w1 = make_float2(0.766044443f, SIGN * 0.642787610f), w2 = make_float2(0.173648178f, SIGN * 0.984807753f),
                 w4 = make_float2(-0.939692621f, SIGN * 0.342020143f);
    v[4] = cmul(v[4], w1);
    v[5] = cmul(v[5], w2);
    v[7] = cmul(v[7], w2);
    v[8] = cmul(v[8], w4);
    // component k2 of the columns gives outputs k2, k2 + 3, k2 + 6
#pragma unroll
    for (int k = 0; k < 3; ++k) dft3<SIGN>(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
    const float2 t[9] = {v[0], v[3], v[6], v[1], v[4], v[7], v[2], v[5], v[8]};
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = t[k];
  } else {
    // R = 2 N, N odd: the prime-factor form (Good 1958), no twiddles between
    static_assert(R == 6 || R == 10, "radix");
    constexpr int N = R / 2;
    float2 t[2][N];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < N; ++b) t[a][b] = v[(N * a + 2 * b) % R];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      if constexpr (N == 3) dft3<SIGN>(t[a][0], t[a][1], t[a][2]);
      else dft5<SIGN>(t[a][0], t[a][1], t[a][2], t[a][3], t[a][4]);
    }
#pragma unroll
    for (int b = 0; b < N; ++b) dft2<SIGN>(t[0][b], t[1][b]);
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = t[k % 2][k % N];
  }
}

// Quotient by a divisor d > 1 without a division: magic = 2^32 / d
// rounded up is exact for numerator x divisor < 2^32 (all FFT indices here
// are below 2^16).  d = 1 (magic 0) means the numerator itself.
__device__ __forceinline__ unsigned quotient(unsigned x, unsigned magic) { return magic ? __umulhi(x, magic) : x; }
__host__ __device__ __forceinline__ unsigned magic_for(unsigned d) { return d > 1 ? 0xFFFFFFFFu / d + 1u : 0u; }

// A transform's twiddle table (n entries) into shared memory, where the
// butterflies read it: a global read in every butterfly stage otherwise.
__device__ __forceinline__ void stage_twiddles(float2* dst, const float2* src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(&src[i]);
}

// One axis' transform plan: the length and its radices, four bits each from
// the first stage up (plan_radices).
struct Axis {
  int n;
  unsigned plan;
};
__device__ __forceinline__ int radix_at(Axis ax, int stage) { return (ax.plan >> (4 * stage)) & 15; }
__device__ __forceinline__ int stages_of(Axis ax) { return (35 - __clz(ax.plan)) >> 2; }

// One Stockham stage of radix R over `nl` lines of length ax.n (ns = the
// product of the radices before it): butterfly (j, l) takes elements
// j + q n/R of line l from `load` and gives elements to `store`.  Lines vary
// fastest over the threads, so with line-fastest layouts every access is
// contiguous.
template <int R, int SIGN, class Load, class Store>
__device__ __forceinline__ void stage_of(int n, int ns, int nl, unsigned nl_magic, const float2* tw, Load load,
                                         Store store) {
  const int bf = n / R, step = bf / ns;
  const unsigned ns_magic = magic_for(unsigned(ns));
  for (int idx = threadIdx.x; idx < nl * bf; idx += blockDim.x) {
    const int j = int(quotient(unsigned(idx), nl_magic)), l = idx - j * nl;
    const int jq = ns == 1 ? j : (step == 1 ? 0 : int(quotient(unsigned(j), ns_magic)));
    const int k = j - jq * ns;
    float2 v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = load(j + q * bf, l);
    if (ns > 1) {
#pragma unroll
      for (int q = 1; q < R; ++q) {
        float2 w = tw[k * q * step];  // k q step < ns R step = n
        if (SIGN > 0) w.y = -w.y;
        v[q] = cmul(v[q], w);
      }
    }
    dft<R, SIGN>(v);
    const int dest = jq * ns * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) store(dest + q * ns, l, v[q]);
  }
}

#define MDB_RADIX_SWITCH(r, CALL) \
  switch (r) {                    \
    case 2: CALL(2); break;       \
    case 3: CALL(3); break;       \
    case 4: CALL(4); break;       \
    case 5: CALL(5); break;       \
    case 6: CALL(6); break;       \
    case 7: CALL(7); break;       \
    case 8: CALL(8); break;       \
    case 9: CALL(9); break;       \
    default: CALL(10); break;     \
  }

// All stages of `nl` lines: the first loads through `load`, the last stores
// through `store` (each given (t, l)), those between go through the two
// buffers, element (t, l) at t * pitch + l.  Ends with a barrier.  Each kind of
// stage is compiled on its own: a block runs few instructions more than once,
// so the fewer it has to fetch the better.
template <int SIGN, class Load, class Store>
__device__ __forceinline__ void transform(Axis ax, int nl, int pitch, const float2* tw, float2* a, float2* b, Load load,
                                          Store store) {
  const int count = stages_of(ax);
  const unsigned nl_magic = magic_for(unsigned(nl));
  const int n = ax.n;
  int ns = radix_at(ax, 0);
  auto from = [&](const float2* p) { return [p, pitch](int t, int l) { return p[t * pitch + l]; }; };
  auto to = [&](float2* p) { return [p, pitch](int t, int l, float2 v) { p[t * pitch + l] = v; }; };
  if (count == 1) {
#define MDB_STAGE(R) stage_of<R, SIGN>(n, 1, nl, nl_magic, tw, load, store)
    MDB_RADIX_SWITCH(ns, MDB_STAGE)
#undef MDB_STAGE
    __syncthreads();
    return;
  }
#define MDB_STAGE(R) stage_of<R, SIGN>(n, 1, nl, nl_magic, tw, load, to(b))
  MDB_RADIX_SWITCH(ns, MDB_STAGE)
#undef MDB_STAGE
  __syncthreads();
  float2 *cur = b, *next = a;
  for (int st = 1; st < count - 1; ++st) {
    const int r = radix_at(ax, st);
#define MDB_STAGE(R) stage_of<R, SIGN>(n, ns, nl, nl_magic, tw, from(cur), to(next))
    MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
    __syncthreads();
    float2* t = cur;
    cur = next;
    next = t;
    ns *= r;
  }
  const int r = radix_at(ax, count - 1);
#define MDB_STAGE(R) stage_of<R, SIGN>(n, ns, nl, nl_magic, tw, from(cur), store)
  MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
  __syncthreads();
}

// ------------------------------------------------------------- splines ----
// Order-5 cardinal B-spline weights and derivatives at fraction w
// (src/reference/forces/bspline.ts:55, the same recursion in f32).
__device__ __forceinline__ void bspline5(float w, float* th, float* dth) {
  float lo[5];
  lo[0] = 1.f - w;
  lo[1] = w;
  lo[2] = 0.f;
  lo[3] = 0.f;
  lo[4] = 0.f;
#pragma unroll
  for (int k = 3; k <= 4; ++k) {
    const float dv = 1.f / (k - 1);
    lo[k - 1] = dv * w * lo[k - 2];
#pragma unroll
    for (int j = 1; j < k - 1; ++j) lo[k - j - 1] = dv * ((w + j) * lo[k - j - 2] + (k - j - w) * lo[k - j - 1]);
    lo[0] = dv * (1.f - w) * lo[0];
  }
  if (dth) {
    dth[0] = -lo[0];
#pragma unroll
    for (int j = 1; j < 5; ++j) dth[j] = lo[j - 1] - lo[j];
  }
#pragma unroll
  for (int j = 0; j < 5; ++j) th[j] = lo[j];
  const float dv = 0.25f;
  th[4] = dv * w * th[3];
#pragma unroll
  for (int j = 1; j < 4; ++j) th[4 - j] = dv * ((w + j) * th[3 - j] + (5 - j - w) * th[4 - j]);
  th[0] = dv * (1.f - w) * th[0];
}

// One axis of an atom's spline from its position: the base mesh index and the
// weights (and derivatives) of its five points.
__device__ __forceinline__ int spline_axis(const SysDev& S, int axis, long long x, long long y, long long z, float* th,
                                           float* dth) {
  const long long u = axis == 0   ? fixed_mul(x, S.umat[0]) + fixed_mul(y, S.umat[1]) + fixed_mul(z, S.umat[2])
                      : axis == 1 ? fixed_mul(y, S.umat[3]) + fixed_mul(z, S.umat[4])
                                  : fixed_mul(z, S.umat[5]);
  const float w = static_cast<float>(static_cast<unsigned int>(u & 0xffffffffll)) * 2.3283064365386963e-10f;
  const int K = S.grid[axis];
  // an atom within a few cells of its box needs a few subtractions, not a
  // 64-bit remainder
  long long b = (u >> 32) - (kPmeOrder - 1);
  if (b < -2ll * K || b >= 3ll * K) b %= K;
  while (b < 0) b += K;
  while (b >= K) b -= K;
  bspline5(w, th, dth);
  return static_cast<int>(b);
}

// ---------------------------------------------------------------- spread --
// The spread reads nothing the list kernels write, so it runs on its own
// stream while the list kernels sort and rebuild: it goes by the slots of a
// snapshot of the list's sorted order that the integrator writes at the end of
// every step (`spread_atom`), never by the order the list kernels are
// rewriting.  A block takes P consecutive slots -- P / 32 super-clusters along
// the space-filling curve, a compact piece of space -- adds their charges into
// a patch of the mesh in shared memory, and adds the patch's nonzero points to
// the grid: an eighth to a quarter of the global atomics of spreading each
// atom's 125 points directly.  The patch holds the block's spline bases
// (unwrapped around its first atom) plus the 5-point stencil; a block whose
// patch would not fit (a cluster torn across a jump of the curve), whose slots
// reach into the next system or that holds a charge of 1,000 e or more (the
// sums' 32-bit halves) spreads directly.  The grid is int64 fixed
// point and every contribution the same value either way, so the grid is the
// same to the bit whatever the order and the route.  What bounds it is a
// block's chain of loads, splines, shared atomics and grid atomics; hence
// short blocks for small engines.  Measured against 128 slots a block from
// 148 blocks up and atomics straight to the grid below: 12k-atom peptide (32
// slots) 13.6 -> 9.2 us, 27k-atom octahedron (64) 24.2 -> 14.4 us, 100k atoms
// (128) 45.6 -> 40.7 us, 64-system ensemble (128) 248 -> 229 us; the
// octahedron at 128 slots took 26.2 us.
constexpr int kPatchPoints = 4096;  // 32 KB in two 32-bit halves
constexpr float kPatchCharge = 1000.f;  // e; any charge there is

// x 2^32 rounded to an integer, as hi 2^20 + lo, for |x| < 1024: both
// roundings are f32 additions of 1.5 2^23 (whose low bits then hold the
// integer), in place of a float-to-int64 conversion at a sixteenth of the f32
// rate.  hi takes the multiple of 2^-12 nearest x, what is left is exact, and
// its rounding to 2^-32 is the whole value's (2^20 is even: ties agree).
__device__ __forceinline__ void split_fixed(float x, int& hi, int& lo) {
  constexpr float kMagic = 12582912.f;  // 1.5 2^23
  const float t = fmaf(x, 4096.f, kMagic);
  const float rest = fmaf(x, 4096.f, -__fsub_rn(t, kMagic));
  hi = __float_as_int(t) - 0x4B400000;
  lo = __float_as_int(fmaf(rest, 1048576.f, kMagic)) - 0x4B400000;
}

template <int P>
__global__ void __launch_bounds__(kThreads) k_spread(Dev d) {
  wait_for_predecessor();
  // the patch's sums in two 32-bit halves (hi 2^20 + lo), so the adds are
  // 32-bit shared atomics: at most P = 128 atoms of less than kPatchCharge add
  // to a point, weights below 1, so |hi| < 2^29 and |lo| <= 2^26
  __shared__ int patch_hi[kPatchPoints], patch_lo[kPatchPoints];
  __shared__ int base[P][3];
  __shared__ float th[P][3][5];
  __shared__ float qs[P];
  __shared__ int sysk[P];
  __shared__ int lo[3], hi[3];
  __shared__ bool heavy;  // some charge is beyond what the halves hold
  const int t = threadIdx.x;
  const int first = blockIdx.x * P;
  if (first >= d.n_slots) return;
  const int last = min(d.n_slots, first + P) - 1;
  // a block may hold the end of one system and the start of the next: then
  // every atom spreads directly into its own system's grid
  const int s = d.slot_sys[first];
  const bool one_system = d.slot_sys[last] == s;
  const int a0 = d.spread_atom[first];
  if (one_system && (a0 < 0 || !sys_active(d, s))) return;  // padding only, or a skipped system
  const SysDev& S = d.sys[s];
  if (t < 3) {
    lo[t] = 1 << 30;
    hi[t] = -(1 << 30);
    heavy = false;
  }
  __syncthreads();
  // splines, a thread per atom and axis (a warp's lanes share the axis)
  for (int w = t; w < 3 * P; w += blockDim.x) {
    const int axis = w / P, k = w - axis * P, gs = first + k;
    const int a = gs <= last ? d.spread_atom[gs] : -1;
    const int st = gs <= last && !one_system ? d.slot_sys[gs] : s;
    const bool live = a >= 0 && sys_active(d, st);
    if (axis == 0) {
      const float q = live ? d.prm_atom[a].w : 0.f;
      if (!(fabsf(q) < kPatchCharge)) heavy = true;
      qs[k] = q;
      sysk[k] = st;
    }
    if (live) {
      float weights[5];
      base[k][axis] = spline_axis(d.sys[st], axis, d.px[a], d.py[a], d.pz[a], weights, nullptr);
#pragma unroll
      for (int i = 0; i < kPmeOrder; ++i) th[k][axis][i] = weights[i];
    }
  }
  __syncthreads();
  if (one_system) {
    // the bases unwrapped around the first atom's, and their range
    for (int w = t; w < 3 * P; w += blockDim.x) {
      const int axis = w / P, k = w - axis * P, K = S.grid[axis];
      const bool live = qs[k] != 0.f;
      int b = 0;
      if (live) {
        const int r = base[0][axis];
        b = base[k][axis];
        if (b - r > K / 2) b -= K;
        if (r - b > K / 2) b += K;
      }
      const int mn = __reduce_min_sync(0xffffffffu, live ? b : 1 << 30);
      const int mx = __reduce_max_sync(0xffffffffu, live ? b : -(1 << 30));
      if ((t & 31) == 0) {
        atomicMin(&lo[axis], mn);
        atomicMax(&hi[axis], mx);
      }
      if (live && k > 0) base[k][axis] = b;
    }
    __syncthreads();
  }
  bool patch = one_system && !heavy;
  int points = 1, ext[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    ext[ax] = hi[ax] - lo[ax] + kPmeOrder;
    patch = patch && hi[ax] >= lo[ax] && ext[ax] <= S.grid[ax];
    if (patch) points *= ext[ax];
    patch = patch && points <= kPatchPoints;
  }
  if (patch) {
    const int ey = ext[1], ez = ext[2], lx = lo[0], ly = lo[1], lz = lo[2];
    for (int i = t; i < points; i += blockDim.x) patch_hi[i] = patch_lo[i] = 0;
    __syncthreads();
    for (int w = t; w < P * kPmeOrder * kPmeOrder; w += blockDim.x) {
      const int k = w / (kPmeOrder * kPmeOrder), r = w - k * kPmeOrder * kPmeOrder;
      const float q = qs[k];
      if (q == 0.f) continue;
      const int ix = r / kPmeOrder, iy = r - ix * kPmeOrder;
      const float wxy = q * th[k][0][ix] * th[k][1][iy];
      const int row = ((base[k][0] - lx + ix) * ey + (base[k][1] - ly + iy)) * ez + (base[k][2] - lz);
#pragma unroll
      for (int iz = 0; iz < kPmeOrder; ++iz) {
        int h, l;
        split_fixed(wxy * th[k][2][iz], h, l);
        atomicAdd(&patch_hi[row + iz], h);
        atomicAdd(&patch_lo[row + iz], l);
      }
    }
    __syncthreads();
    const unsigned plane_magic = magic_for(unsigned(ey * ez)), row_magic = magic_for(unsigned(ez));
    const int Kx = S.grid[0], Ky = S.grid[1], Kz = S.grid[2];
    unsigned long long* grid = d.qgrid + S.grid_off;
    // the patch's first point, turned into the mesh (its unwrapped base lies
    // within half a mesh of one in it): no point is then a second turn away,
    // however short the axis and whether or not the first atom has a charge
    const int ox = lx + (lx < 0 ? Kx : (lx >= Kx ? -Kx : 0)), oy = ly + (ly < 0 ? Ky : (ly >= Ky ? -Ky : 0)),
              oz = lz + (lz < 0 ? Kz : (lz >= Kz ? -Kz : 0));
    for (int i = t; i < points; i += blockDim.x) {
      const long long v = static_cast<long long>(patch_hi[i]) * (1ll << 20) + patch_lo[i];
      if (!v) continue;
      const int px = int(quotient(unsigned(i), plane_magic)), rem = i - px * ey * ez;
      const int py = int(quotient(unsigned(rem), row_magic)), pz = rem - py * ez;
      const int gx = ox + px - (ox + px >= Kx ? Kx : 0), gy = oy + py - (oy + py >= Ky ? Ky : 0),
                gz = oz + pz - (oz + pz >= Kz ? Kz : 0);
      add_fixed64(grid + (static_cast<long long>(gx) * Ky + gy) * Kz + gz, v);
    }
  } else {
    // the direct spread of each atom's 125 points, into its own system's grid
    for (int w = t; w < P * kPmeOrder * kPmeOrder; w += blockDim.x) {
      const int k = w / (kPmeOrder * kPmeOrder), r = w - k * kPmeOrder * kPmeOrder;
      const float q = qs[k];
      if (q == 0.f) continue;
      const SysDev& Sk = d.sys[sysk[k]];
      const int Kx = Sk.grid[0], Ky = Sk.grid[1], Kz = Sk.grid[2];
      const int ix = r / kPmeOrder, iy = r - ix * kPmeOrder;
      int gx = (base[k][0] + ix) % Kx, gy = (base[k][1] + iy) % Ky;
      if (gx < 0) gx += Kx;
      if (gy < 0) gy += Ky;
      const float wxy = q * th[k][0][ix] * th[k][1][iy];
      unsigned long long* row = d.qgrid + Sk.grid_off + (static_cast<long long>(gx) * Ky + gy) * Kz;
#pragma unroll
      for (int iz = 0; iz < kPmeOrder; ++iz) {
        int gz = (base[k][2] + iz) % Kz;
        if (gz < 0) gz += Kz;
        add_fixed(&row[gz], wxy * th[k][2][iz]);
      }
    }
  }
}

// ---------------------------------------------------------------- passes --
// A mesh as the passes see it: the engine's tables of one system, or the
// allocation-free path's.
struct Mesh {
  Axis x, y, z;
  int kzh;  // Kz / 2 + 1
  unsigned long long* charge;  // [Kx][Ky][Kz], 2^32 fixed point; cleared as it is read
  float2* spectrum;            // [Kx][Ky][kzh]
  float* potential;            // [Kx][Ky][Kz]
  const float2 *twx, *twy, *twz;
};

__device__ __forceinline__ Mesh mesh_of(const Dev& d, const SysDev& S) {
  Mesh m;
  m.x = {S.grid[0], S.plan[0]};
  m.y = {S.grid[1], S.plan[1]};
  m.z = {S.grid[2], S.plan[2]};
  m.kzh = S.kzh;
  m.charge = d.qgrid + S.grid_off;
  m.spectrum = d.cgrid + S.cgrid_off;
  m.potential = d.phi + S.grid_off;
  m.twx = d.twiddles + S.tw_off[0];
  m.twy = d.twiddles + S.tw_off[1];
  m.twz = d.twiddles + S.tw_off[2];
  return m;
}

// The z transforms take real lines two at a time: lines y = 2p and 2p + 1 of
// an x-plane are the real and the imaginary part of one complex line, whose
// transform Z gives both: (Z_k + conj Z_-k) / 2 and (Z_k - conj Z_-k) / 2i.
// The pairs are counted inside the plane (an odd Ky leaves the last line
// alone), whichever kernel runs them, so all give the same bits.
__device__ __forceinline__ float2 line_of_pair(float2 a, float2 b, bool odd) {  // a = Z_k, b = Z_-k
  return odd ? make_float2(0.5f * __fadd_rn(a.y, b.y), 0.5f * __fsub_rn(b.x, a.x))
             : make_float2(0.5f * __fadd_rn(a.x, b.x), 0.5f * __fsub_rn(a.y, b.y));
}
// The inverse: element t of the complex line of two half spectra.  Elements
// 0 and Kz/2 of a real line's spectrum are real; what rounding left in their
// imaginary parts would run into the other line.
template <class Half>
__device__ __forceinline__ float2 pair_of_lines(int Kz, int t, bool second, Half half) {
  const int k = 2 * t <= Kz ? t : Kz - t;
  float2 a = half(0, k), b = second ? half(1, k) : make_float2(0.f, 0.f);
  if (t == 0 || 2 * t == Kz) a.y = b.y = 0.f;
  if (k != t) {
    a.y = -a.y;
    b.y = -b.y;
  }
  return make_float2(__fsub_rn(a.x, b.y), __fadd_rn(a.y, b.x));
}

// Pitches and sizes of the plane passes' two shared buffers: z lines
// [Kz][pairs] (an odd pitch keeps the charge loads' bank conflicts at two), y
// lines [Ky][kzh].
__host__ __device__ __forceinline__ int pair_pitch(int lines) { return ((lines + 1) / 2) | 1; }
__host__ __device__ __forceinline__ int plane_buffer(int Ky, int Kz) {
  const int z = Kz * pair_pitch(Ky), y = Ky * (Kz / 2 + 1);
  return z > y ? z : y;
}

// Charges of `lines` consecutive z lines (from an even one of the plane) into
// paired complex lines, clearing the grid ("consumer clears": the next spread
// starts from zero).
__device__ __forceinline__ void load_charges(unsigned long long* grid, int lines, int Kz, int pitch, float2* a) {
  const unsigned kz_magic = magic_for(unsigned(Kz));
  float* flat = reinterpret_cast<float*>(a);
  const int total = lines * Kz;
  // four loads in flight per thread before any is used
  for (int i0 = threadIdx.x; i0 < total; i0 += 4 * blockDim.x) {
    long long v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * blockDim.x;
      v[u] = i < total ? static_cast<long long>(__ldcg(&grid[i])) : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < total) {
        const int y = int(quotient(unsigned(i), kz_magic)), z = i - y * Kz;
        flat[(z * pitch + (y >> 1)) * 2 + (y & 1)] = from_fixed(v[u]);
        grid[i] = 0ull;
      }
    }
  }
  if (lines & 1)
    for (int z = threadIdx.x; z < Kz; z += blockDim.x) a[z * pitch + (lines >> 1)].y = 0.f;
}

// Real lines out of paired complex lines.
__device__ __forceinline__ void store_potential(float* out, int lines, int Kz, int pitch, const float2* a) {
  const unsigned kz_magic = magic_for(unsigned(Kz));
  const float* flat = reinterpret_cast<const float*>(a);
  for (int i = threadIdx.x; i < lines * Kz; i += blockDim.x) {
    const int y = int(quotient(unsigned(i), kz_magic)), z = i - y * Kz;
    out[i] = flat[(z * pitch + (y >> 1)) * 2 + (y & 1)];
  }
}

// Whole x-planes: z and y of one plane by one CTA, so a transform in one
// direction is two launches (with the x pass) and each has a plane of work.
// What bounds them is the chain of one CTA (a load, four stages, four
// barriers, a store), not bandwidth: 50^3 moves 2 MB.  Two real lines to a
// complex one halve the z stages; radices up to 10 make most axes two stages;
// the y transform's first stage separates the pairs as it loads and its last
// stores to global memory, so nothing is copied between.  Measured with the x
// pass against radices up to 5, lines one at a time and copies between the
// axes: 50^3 27.7 -> 21.2 us, 60 x 54 x 48 30.6 -> 21.4 us, 81^3 54 -> 29 us,
// the 64-system ensemble's meshes 274 -> 92 us.
__device__ __forceinline__ void plane_forward(const Mesh& m, int x, float2* smem) {
  const int Ky = m.y.n, Kz = m.z.n, kzh = m.kzh, pitch = pair_pitch(Ky), size = plane_buffer(Ky, Kz);
  float2 *a = smem, *b = smem + size, *twz = smem + 2 * size, *twy = twz + Kz;
  stage_twiddles(twz, m.twz, Kz);
  stage_twiddles(twy, m.twy, Ky);
  load_charges(m.charge + static_cast<long long>(x) * Ky * Kz, Ky, Kz, pitch, a);
  __syncthreads();
  // an even number of stages comes back to the first buffer
  const bool swapped = stages_of(m.z) & 1;
  transform<-1>(m.z, (Ky + 1) / 2, pitch, twz, a, b, [&](int t, int l) { return a[t * pitch + l]; },
                [&](int t, int l, float2 v) { (swapped ? b : a)[t * pitch + l] = v; });
  const float2* Z = swapped ? b : a;
  float2 *free0 = swapped ? a : b, *free1 = swapped ? b : a;
  float2* out = m.spectrum + static_cast<long long>(x) * Ky * kzh;
  transform<-1>(m.y, kzh, kzh, twy, free1, free0,
                [&](int y, int k) {
                  const int p = y >> 1;
                  return line_of_pair(Z[k * pitch + p], Z[(k ? Kz - k : 0) * pitch + p], y & 1);
                },
                [&](int y, int k, float2 v) { out[y * kzh + k] = v; });
}

__device__ __forceinline__ void plane_inverse(const Mesh& m, int x, float2* smem) {
  const int Ky = m.y.n, Kz = m.z.n, kzh = m.kzh, pitch = pair_pitch(Ky), size = plane_buffer(Ky, Kz);
  float2 *a = smem, *b = smem + size, *twz = smem + 2 * size, *twy = twz + Kz;
  stage_twiddles(twz, m.twz, Kz);
  stage_twiddles(twy, m.twy, Ky);
  const float2* in = m.spectrum + static_cast<long long>(x) * Ky * kzh;
  __syncthreads();
  const bool swapped = stages_of(m.y) & 1;
  transform<+1>(m.y, kzh, kzh, twy, a, b, [&](int y, int k) { return __ldcg(&in[y * kzh + k]); },
                [&](int y, int k, float2 v) { (swapped ? b : a)[y * kzh + k] = v; });
  const float2* Y = swapped ? b : a;
  float2 *free0 = swapped ? a : b, *free1 = swapped ? b : a;
  float2* R = stages_of(m.z) & 1 ? free0 : free1;
  transform<+1>(m.z, (Ky + 1) / 2, pitch, twz, free1, free0,
                [&](int t, int p) {
                  return pair_of_lines(Kz, t, 2 * p + 1 < Ky, [&](int h, int k) { return Y[(2 * p + h) * kzh + k]; });
                },
                [&](int t, int p, float2 v) { R[t * pitch + p] = v; });
  store_potential(m.potential + static_cast<long long>(x) * Ky * Kz, Ky, Kz, pitch, R);
}

// z and y passes of their own, for planes that do not fit shared memory: lines
// [line0, line0 + lines) of the mesh, an even number from an even line of
// one plane (or the rest of it); a strip of `nk` kz columns of an x-plane.
__device__ __forceinline__ void z_forward(const Mesh& m, int line0, int lines, float2* smem) {
  const int Kz = m.z.n, kzh = m.kzh, pitch = pair_pitch(lines);
  float2 *a = smem, *b = smem + Kz * pitch, *tw = smem + 2 * Kz * pitch;
  stage_twiddles(tw, m.twz, Kz);
  load_charges(m.charge + static_cast<long long>(line0) * Kz, lines, Kz, pitch, a);
  __syncthreads();
  const bool swapped = stages_of(m.z) & 1;
  transform<-1>(m.z, (lines + 1) / 2, pitch, tw, a, b, [&](int t, int l) { return a[t * pitch + l]; },
                [&](int t, int l, float2 v) { (swapped ? b : a)[t * pitch + l] = v; });
  const float2* Z = swapped ? b : a;
  float2* out = m.spectrum + static_cast<long long>(line0) * kzh;
  for (int i = threadIdx.x; i < lines * kzh; i += blockDim.x) {
    const int y = i / kzh, k = i - y * kzh, p = y >> 1;
    out[i] = line_of_pair(Z[k * pitch + p], Z[(k ? Kz - k : 0) * pitch + p], y & 1);
  }
}

__device__ __forceinline__ void z_inverse(const Mesh& m, int line0, int lines, float2* smem) {
  const int Kz = m.z.n, kzh = m.kzh, pitch = pair_pitch(lines);
  float2 *a = smem, *b = smem + Kz * pitch, *tw = smem + 2 * Kz * pitch;
  stage_twiddles(tw, m.twz, Kz);
  const float2* in = m.spectrum + static_cast<long long>(line0) * kzh;
  __syncthreads();
  float2* R = stages_of(m.z) & 1 ? b : a;
  transform<+1>(m.z, (lines + 1) / 2, pitch, tw, a, b,
                [&](int t, int p) {
                  return pair_of_lines(Kz, t, 2 * p + 1 < lines,
                                       [&](int h, int k) { return __ldcg(&in[(2 * p + h) * kzh + k]); });
                },
                [&](int t, int p, float2 v) { R[t * pitch + p] = v; });
  store_potential(m.potential + static_cast<long long>(line0) * Kz, lines, Kz, pitch, R);
}

template <int SIGN>
__device__ __forceinline__ void y_pass(const Mesh& m, int x, int kz0, int nk, float2* smem) {
  const int Ky = m.y.n, kzh = m.kzh;
  float2 *a = smem, *b = smem + nk * Ky, *tw = smem + 2 * nk * Ky;
  stage_twiddles(tw, m.twy, Ky);
  float2* base = m.spectrum + static_cast<long long>(x) * Ky * kzh + kz0;
  __syncthreads();
  transform<SIGN>(m.y, nk, nk, tw, a, b, [&](int y, int l) { return base[static_cast<long long>(y) * kzh + l]; },
                  [&](int y, int l, float2 v) { base[static_cast<long long>(y) * kzh + l] = v; });
}

// The x pass: `nk` lines at (y, kz0 ..), forward, each element through
// `factor(mx, l, v)`, inverse.  The inverse runs the radices backwards, so its
// first butterflies take exactly the elements the forward transform's last
// ones give: those two stages and the factor happen in registers, and a
// two-stage axis makes three passes with two barriers in all, loading and
// storing global memory directly.
template <class Factor>
__device__ __forceinline__ void x_pass(const Mesh& m, int y, int kz0, int nk, float2* smem, Factor factor) {
  const int Kx = m.x.n, count = stages_of(m.x);
  float2 *a = smem, *b = smem + nk * Kx, *tw = smem + 2 * nk * Kx;
  stage_twiddles(tw, m.twx, Kx);
  const long long stride = static_cast<long long>(m.y.n) * m.kzh;
  float2* base = m.spectrum + static_cast<long long>(y) * m.kzh + kz0;
  const unsigned nk_magic = magic_for(unsigned(nk));
  __syncthreads();
  auto load = [&](int t, int l) { return __ldcg(&base[t * stride + l]); };
  auto save = [&](int t, int l, float2 v) { base[t * stride + l] = v; };
  auto from = [&](const float2* p) { return [p, nk](int t, int l) { return p[t * nk + l]; }; };
  auto to = [&](float2* p) { return [p, nk](int t, int l, float2 v) { p[t * nk + l] = v; }; };
  auto swap = [&]() {
    float2* t = a;
    a = b;
    b = t;
  };
  // forward, up to the last stage: from global memory into b, then a to b
  int ns = 1;
  for (int st = 0; st < count - 1; ++st) {
    const int r = radix_at(m.x, st);
    if (st == 0) {
#define MDB_STAGE(R) stage_of<R, -1>(Kx, 1, nk, nk_magic, tw, load, to(b))
      MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
    } else {
#define MDB_STAGE(R) stage_of<R, -1>(Kx, ns, nk, nk_magic, tw, from(a), to(b))
      MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
    }
    __syncthreads();
    swap();
    ns *= r;
  }
  // the forward transform's last butterflies, the factor, the inverse's first
  const int turn = radix_at(m.x, count - 1);
  auto middle = [&](auto radix, auto in, auto out) {
    constexpr int R = decltype(radix)::value;
    const int bf = Kx / R;
    for (int idx = threadIdx.x; idx < nk * bf; idx += blockDim.x) {
      const int k = int(quotient(unsigned(idx), nk_magic)), l = idx - k * nk;
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = in(k + q * bf, l);
      if (bf > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[k * q]);
      }
      dft<R, -1>(v);
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = factor(k + q * bf, l, v[q]);
      dft<R, +1>(v);
#pragma unroll
      for (int q = 0; q < R; ++q) out(k * R + q, l, v[q]);
    }
  };
  if (count == 1) {
#define MDB_TURN(R) middle(std::integral_constant<int, R>{}, load, save)
    MDB_RADIX_SWITCH(turn, MDB_TURN)
#undef MDB_TURN
    __syncthreads();
    return;
  }
#define MDB_TURN(R) middle(std::integral_constant<int, R>{}, from(a), to(b))
  MDB_RADIX_SWITCH(turn, MDB_TURN)
#undef MDB_TURN
  __syncthreads();
  ns = turn;
  for (int st = count - 2; st >= 0; --st) {
    swap();
    const int r = radix_at(m.x, st);
    if (st == 0) {
#define MDB_STAGE(R) stage_of<R, +1>(Kx, ns, nk, nk_magic, tw, from(a), save)
      MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
    } else {
#define MDB_STAGE(R) stage_of<R, +1>(Kx, ns, nk, nk_magic, tw, from(a), to(b))
      MDB_RADIX_SWITCH(r, MDB_STAGE)
#undef MDB_STAGE
    }
    __syncthreads();
    ns *= r;
  }
}

// ------------------------------------------------ the Ewald convolution ---
// The Ewald influence function (pme-convolve.wgsl:34; pme.ts:160-209) at
// mesh index (mx, my, kz) of the half spectrum, mb the signed y index; the
// wave vector and its square come back for the virial.  0 at the origin.
// Written with explicit roundings so the table and the energy variant agree
// to the bit.
__device__ __forceinline__ float influence(const SysDev& S, const float* modx, const float* mody, const float* modz,
                                           int Kx, int mx, int mb, int my, int kz, float& kx, float& ky, float& kzv,
                                           float& k2) {
  if (mx == 0 && my == 0 && kz == 0) return 0.f;
  const float two_pi = 6.283185307179586f;
  const float* M = S.inv_f;
  const float ma = static_cast<float>(mx <= Kx / 2 ? mx : mx - Kx), fb = static_cast<float>(mb),
              mc = static_cast<float>(kz);  // kz <= Kz/2 on the half spectrum
  kx = __fmul_rn(two_pi, __fmul_rn(ma, M[0]));
  ky = __fmul_rn(two_pi, fmaf(fb, M[4], __fmul_rn(ma, M[3])));
  kzv = __fmul_rn(two_pi, fmaf(mc, M[8], fmaf(fb, M[7], __fmul_rn(ma, M[6]))));
  k2 = fmaf(kzv, kzv, fmaf(ky, ky, __fmul_rn(kx, kx)));
  const float den = __fmul_rn(__fmul_rn(__fmul_rn(k2, modx[mx]), mody[my]), modz[kz]);
  return __fdiv_rn(__fmul_rn(S.pme_pref, expf(__fmul_rn(k2, S.exp_scale))), den);
}

// The influence function of every x-pass work item of system `s` (all
// systems: s < 0), element (mx, l) at mx * lines + l as the x pass reads it.
// Run after every change of a box.
__global__ void __launch_bounds__(kThreads) k_influence(Dev d, int s) {
  const FftWork w = d.fft_x[blockIdx.x];
  if (s >= 0 && w.sys != s) return;
  const SysDev& S = d.sys[w.sys];
  const int Kx = S.grid[0], Ky = S.grid[1];
  const float* modx = d.moduli + S.mod_off;
  const float* mody = modx + Kx;
  const float* modz = mody + Ky;
  const int my = w.a, mb = my <= Ky / 2 ? my : my - Ky;
  float* table = d.influence + static_cast<long long>(blockIdx.x) * d.influence_stride;
  for (int i = threadIdx.x; i < w.n * Kx; i += blockDim.x) {
    const int mx = i / w.n, l = i - mx * w.n;
    float kx, ky, kzv, k2;
    table[i] = influence(S, modx, mody, modz, Kx, mx, mb, my, w.b + l, kx, ky, kzv, k2);
  }
}

constexpr int kXThreads = 128;  // eight lines of 50 points are 80 or 40 butterflies a stage

// The block's sums of `val`, in a fixed order in FP64 (deterministic), to out(c, total).
template <int N, class Out>
__device__ __forceinline__ void block_sums(double* val, Out out) {
  __shared__ double partial[N][kXThreads / 32];
#pragma unroll
  for (int c = 0; c < N; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) val[c] += __shfl_xor_sync(0xffffffffu, val[c], o);
    if ((threadIdx.x & 31) == 0) partial[c][threadIdx.x >> 5] = val[c];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double total = 0.0;
    for (int k = 0; k < int(blockDim.x >> 5); ++k) total += partial[threadIdx.x][k];
    out(int(threadIdx.x), total);
  }
}

template <bool ENERGY>
__global__ void __launch_bounds__(kXThreads) k_fft_x_convolve(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_x[blockIdx.x];
  if (!sys_active(d, w.sys)) return;  // the whole block: before any barrier
  const SysDev& S = d.sys[w.sys];
  const Mesh m = mesh_of(d, S);
  const int my = w.a, nk = w.n;
  // the force variant (every MD step) reads the influence function from the
  // table k_influence fills at every box change; the energy variant needs the
  // wave vectors for the virial and evaluates it here, the same function
  const float* table = d.influence + static_cast<long long>(blockIdx.x) * d.influence_stride;
  double sums[7] = {0, 0, 0, 0, 0, 0, 0};  // energy, virial xx yy zz xy xz yz
  x_pass(m, my, w.b, nk, smem, [&](int mx, int l, float2 v) {
    float f;
    if (ENERGY) {
      const int Kx = m.x.n, Ky = m.y.n, Kz = m.z.n, kz = w.b + l, mb = my <= Ky / 2 ? my : my - Ky;
      const float* modx = d.moduli + S.mod_off;
      float kx = 0.f, ky = 0.f, kzv = 0.f, k2 = 1.f;
      f = influence(S, modx, modx + Kx, modx + Kx + Ky, Kx, mx, mb, my, kz, kx, ky, kzv, k2);
      const double weight = (kz == 0 || (2 * kz == Kz)) ? 1.0 : 2.0;
      const double ek =
          weight * static_cast<double>(f) * (static_cast<double>(v.x) * v.x + static_cast<double>(v.y) * v.y);
      // -dE_k/d eps_ab = E_k (delta_ab - 2 k_a k_b (1/k^2 + 1/(4 alpha^2)))
      const double c = 2.0 * (1.0 / static_cast<double>(k2) - static_cast<double>(S.exp_scale));
      const double ka = kx, kb = ky, kc = kzv;
      sums[0] += ek;
      sums[1] += ek * (1.0 - c * ka * ka);
      sums[2] += ek * (1.0 - c * kb * kb);
      sums[3] += ek * (1.0 - c * kc * kc);
      sums[4] -= ek * c * ka * kb;
      sums[5] -= ek * c * ka * kc;
      sums[6] -= ek * c * kb * kc;
    } else {
      f = __ldg(&table[mx * nk + l]);
    }
    const float g = 2.f * f;
    return make_float2(__fmul_rn(v.x, g), __fmul_rn(v.y, g));
  });
  if (ENERGY) {
    block_sums<7>(sums, [&](int c, double total) {
      if (c == 0) d.mesh_partial[blockIdx.x] = total;
      else d.mesh_virial[blockIdx.x * 6 + c - 1] = total;
    });
  }
}

constexpr int kPlaneThreads = 256;

__global__ void __launch_bounds__(kPlaneThreads) k_fft_zy_forward(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_p[blockIdx.x];
  if (!sys_active(d, w.sys)) return;  // the whole block: before any barrier
  plane_forward(mesh_of(d, d.sys[w.sys]), w.a, smem);
}

__global__ void __launch_bounds__(kPlaneThreads) k_fft_yz_inverse(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_p[blockIdx.x];
  if (!sys_active(d, w.sys)) return;
  plane_inverse(mesh_of(d, d.sys[w.sys]), w.a, smem);
}

__global__ void __launch_bounds__(kThreads) k_fft_z_forward(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_z[blockIdx.x];
  if (!sys_active(d, w.sys)) return;
  z_forward(mesh_of(d, d.sys[w.sys]), w.a, w.n, smem);
}

template <int SIGN>
__global__ void __launch_bounds__(kThreads) k_fft_y(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_y[blockIdx.x];
  if (!sys_active(d, w.sys)) return;
  y_pass<SIGN>(mesh_of(d, d.sys[w.sys]), w.a, w.b, w.n, smem);
}

__global__ void __launch_bounds__(kThreads) k_fft_z_inverse(Dev d) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const FftWork w = d.fft_z[blockIdx.x];
  if (!sys_active(d, w.sys)) return;
  z_inverse(mesh_of(d, d.sys[w.sys]), w.a, w.n, smem);
}

// ---------------------------------------------------------------- gather --
// A block of 32 atoms: their splines first, a warp to an axis; then a warp to
// each of the five x planes of the stencil, lanes atoms, with the plane's 25
// loads in flight together; then the five partial sums in a fixed order.  A
// thread per atom walking its 125 points left the kernel waiting on loads with
// few warps to hide them (12k-atom peptide 6.5 -> 5.2 us, 100k atoms 21.6 ->
// 18.9 us).
constexpr int kGatherAtoms = 32;
constexpr int kGatherThreads = 32 * kPmeOrder;

struct GatherTable {
  int base[3][kGatherAtoms];
  float th[3][5][kGatherAtoms], dth[3][5][kGatherAtoms];
  float part[kPmeOrder][3][kGatherAtoms];
};

// `live`: whether this lane's atom (the same in every warp) has a charge; x,
// y, z its position.  Returns true in warp 0 for the live atoms, with the
// gradient of the potential along the mesh axes.
__device__ __forceinline__ bool gather_block(GatherTable& t, bool live, const SysDev& S, const float* grid, long long x,
                                             long long y, long long z, float& ga, float& gb, float& gc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (live && warp < 3) {
    float th[5], dth[5];
    t.base[warp][lane] = spline_axis(S, warp, x, y, z, th, dth);
#pragma unroll
    for (int i = 0; i < kPmeOrder; ++i) {
      t.th[warp][i][lane] = th[i];
      t.dth[warp][i][lane] = dth[i];
    }
  }
  __syncthreads();
  ga = gb = gc = 0.f;
  if (live) {
    const int Kx = S.grid[0], Ky = S.grid[1], Kz = S.grid[2];
    int gx = t.base[0][lane] + warp;
    if (gx >= Kx) gx -= Kx;
    const int by = t.base[1][lane], bz = t.base[2][lane];
    int gz[5];
#pragma unroll
    for (int iz = 0; iz < kPmeOrder; ++iz) {
      gz[iz] = bz + iz;
      if (gz[iz] >= Kz) gz[iz] -= Kz;
    }
    float p[5][5];
#pragma unroll
    for (int iy = 0; iy < kPmeOrder; ++iy) {
      int gy = by + iy;
      if (gy >= Ky) gy -= Ky;
      const float* row = grid + (static_cast<long long>(gx) * Ky + gy) * Kz;
#pragma unroll
      for (int iz = 0; iz < kPmeOrder; ++iz) p[iy][iz] = row[gz[iz]];
    }
    const float wx = t.th[0][warp][lane], dx = t.dth[0][warp][lane];
#pragma unroll
    for (int iy = 0; iy < kPmeOrder; ++iy) {
      float along = 0.f, slope = 0.f;
#pragma unroll
      for (int iz = 0; iz < kPmeOrder; ++iz) {
        along = fmaf(p[iy][iz], t.th[2][iz][lane], along);
        slope = fmaf(p[iy][iz], t.dth[2][iz][lane], slope);
      }
      const float wy = t.th[1][iy][lane], dy = t.dth[1][iy][lane];
      ga = fmaf(along, __fmul_rn(dx, wy), ga);
      gb = fmaf(along, __fmul_rn(wx, dy), gb);
      gc = fmaf(slope, __fmul_rn(wx, wy), gc);
    }
    if (warp > 0) {
      t.part[warp][0][lane] = ga;
      t.part[warp][1][lane] = gb;
      t.part[warp][2][lane] = gc;
    }
  }
  __syncthreads();
  if (!live || warp > 0) return false;
#pragma unroll
  for (int w = 1; w < kPmeOrder; ++w) {
    ga = __fadd_rn(ga, t.part[w][0][lane]);
    gb = __fadd_rn(gb, t.part[w][1][lane]);
    gc = __fadd_rn(gc, t.part[w][2][lane]);
  }
  return true;
}

// F_v = -q sum_u (dE/du_u) K_u M[v][u]  (pme.ts:252-259)
__device__ __forceinline__ float3 mesh_force(const SysDev& S, float q, float ga, float gb, float gc) {
  const float* U = S.umat_f;
  return make_float3(__fmul_rn(-q, fmaf(gc, U[2], fmaf(gb, U[1], __fmul_rn(ga, U[0])))),
                     __fmul_rn(-q, fmaf(gc, U[5], fmaf(gb, U[4], __fmul_rn(ga, U[3])))),
                     __fmul_rn(-q, fmaf(gc, U[8], fmaf(gb, U[7], __fmul_rn(ga, U[6])))));
}

__global__ void __launch_bounds__(kGatherThreads) k_gather(Dev d) {
  wait_for_predecessor();
  __shared__ GatherTable table;
  const int gs = blockIdx.x * kGatherAtoms + (threadIdx.x & 31);  // n_slots is a multiple of 32
  const int a = d.order[gs], s = d.slot_sys[gs];
  const float q = a >= 0 ? d.prm[gs].w : 0.f;
  const bool live = q != 0.f && sys_active(d, s);
  const SysDev& S = d.sys[s];
  float ga, gb, gc;
  if (!gather_block(table, live, S, d.phi + S.grid_off, live ? d.px[a] : 0, live ? d.py[a] : 0, live ? d.pz[a] : 0, ga,
                    gb, gc))
    return;
  const float3 f = mesh_force(S, q, ga, gb, gc);
  add_fixed(&d.fx[gs], f.x);
  add_fixed(&d.fy[gs], f.y);
  add_fixed(&d.fz[gs], f.z);
}

}  // namespace

// Shared-memory bytes of one work item of each transform pass.
int plane_smem(int Ky, int Kz) { return (2 * plane_buffer(Ky, Kz) + Ky + Kz) * int(sizeof(float2)); }
int z_smem(int lines, int Kz) { return (2 * pair_pitch(lines) + 1) * Kz * int(sizeof(float2)); }
int strip_smem(int lines, int n) { return (2 * lines + 1) * n * int(sizeof(float2)); }

// Every transform kernel may use up to `bytes` of dynamic shared memory (the
// launches ask for their own engine's size): called once per engine with the
// device's limit, so engines of different meshes do not disturb one another.
int allow_pme_smem(int bytes) {
  cudaError_t err = cudaSuccess;
  auto allow = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) err = e;
  };
  allow(k_fft_zy_forward);
  allow(k_fft_yz_inverse);
  allow(k_fft_z_forward);
  allow(k_fft_z_inverse);
  allow(k_fft_x_convolve<true>);
  allow(k_fft_x_convolve<false>);
  allow(k_fft_y<-1>);
  allow(k_fft_y<+1>);
  return err == cudaSuccess ? 0 : 1;
}

void launch_pme_spread(const Dev& d, cudaStream_t st) {
  if (d.n_fft_z == 0) return;
  // the most slots per block that still give every SM two blocks: compact
  // patches share more points, short blocks have short chains
  const int n = d.n_slots;
  auto blocks = [n](int p) { return (n + p - 1) / p; };
  if (blocks(128) >= 2 * 148) launch_chained(k_spread<128>, blocks(128), kThreads, 0, st, d);
  else if (blocks(64) >= 2 * 148) launch_chained(k_spread<64>, blocks(64), kThreads, 0, st, d);
  else launch_chained(k_spread<32>, blocks(32), kThreads, 0, st, d);
}

void launch_pme_fft(const Dev& d, bool energy, cudaStream_t st) {
  if (d.n_fft_z == 0) return;
  if (d.fft_planes) launch_chained(k_fft_zy_forward, d.n_fft_p, kPlaneThreads, d.smem_p, st, d);
  else {
    launch_chained(k_fft_z_forward, d.n_fft_z, kThreads, d.smem_z, st, d);
    launch_chained(k_fft_y<-1>, d.n_fft_y, kThreads, d.smem_y, st, d);
  }
  if (energy) launch_chained(k_fft_x_convolve<true>, d.n_fft_x, kXThreads, d.smem_x, st, d);
  else launch_chained(k_fft_x_convolve<false>, d.n_fft_x, kXThreads, d.smem_x, st, d);
  if (d.fft_planes) launch_chained(k_fft_yz_inverse, d.n_fft_p, kPlaneThreads, d.smem_p, st, d);
  else {
    launch_chained(k_fft_y<+1>, d.n_fft_y, kThreads, d.smem_y, st, d);
    launch_chained(k_fft_z_inverse, d.n_fft_z, kThreads, d.smem_z, st, d);
  }
}

void launch_influence(const Dev& d, int s, cudaStream_t st) {
  if (d.n_fft_x == 0) return;
  k_influence<<<d.n_fft_x, kThreads, 0, st>>>(d, s);
}

void launch_pme_gather(const Dev& d, cudaStream_t st) {
  if (d.n_fft_z == 0) return;
  launch_chained(k_gather, d.n_slots / kGatherAtoms, kGatherThreads, 0, st, d);
}

void launch_pme(const Dev& d, bool energy, cudaStream_t st) {
  launch_pme_spread(d, st);
  launch_pme_fft(d, energy, st);
  launch_pme_gather(d, st);
}

}  // namespace mdb

// ===========================================================================
// Reciprocal-space PME with no allocation: for callers that cannot allocate
// device memory themselves -- code running inside another framework's memory
// pool, a host whose only device memory is what its own allocator hands out,
// or a real-time loop that forbids allocation after start-up.  The caller
// passes its own device buffers for the inputs and outputs; every
// intermediate (charge grid, half spectrum, potential, B-spline moduli,
// twiddles, energy partials) lives in one file-scope device array of fixed
// size, so this path never calls cudaMalloc, cudaFree or any allocating
// library routine.
//
// Limits: at most kNoAllocMaxMeshPoints mesh points (64^3), kNoAllocMaxAxis
// points per axis and at least kPmeOrder.  Every call uses the same array and leaves
// its contents behind; the charge grid is cleared at the start of each call.
// Two calls whose device work overlaps (different streams, or different host
// threads on one device) race on the array and must be serialised by the
// caller.
// ===========================================================================
namespace mdb {
namespace {

constexpr long long kNoAllocMaxMeshPoints = 64ll * 64 * 64;
constexpr int kNoAllocMaxAxis = 128;
// planes up to this size are transformed whole: what a block may use without
// asking for more (64 x 64 needs 35 KB)
constexpr int kNoAllocPlaneSmem = 48 * 1024;
constexpr int kNoAllocMaxPartials = kNoAllocMaxAxis * ((kNoAllocMaxAxis / 2 + 1 + kFftTile - 1) / kFftTile);

// Byte offsets of the pieces inside the scratch array.
constexpr size_t kNaGrid = 0;                                           // int64 x K
constexpr size_t kNaSpectrum = kNaGrid + 8 * kNoAllocMaxMeshPoints;     // float2 x Kh (<= K)
constexpr size_t kNaPotential = kNaSpectrum + 8 * kNoAllocMaxMeshPoints;  // f32 x K
constexpr size_t kNaModuli = kNaPotential + 4 * kNoAllocMaxMeshPoints;  // f32 x 3 axes
constexpr size_t kNaTwiddles = kNaModuli + 4 * 3 * kNoAllocMaxAxis;     // float2 x 3 axes
constexpr size_t kNaPartials = kNaTwiddles + 8 * 3 * kNoAllocMaxAxis;   // f64 per x-pass CTA
constexpr size_t kNaBytes = kNaPartials + 8 * kNoAllocMaxPartials;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

struct NaPtrs {
  unsigned long long* grid;
  float2* spectrum;
  float* potential;
  float* moduli;
  float2* twiddles;
  double* partials;
};

// Twiddles exp(-2 pi i j / K) and moduli |b(m)|^2 of the order-5 spline
// (bspline.ts:102) of each axis, computed on the device in FP64 by the first
// three blocks, one sine and cosine a point; and the charge grid cleared,
// because the array keeps the previous call's contents.
__global__ void __launch_bounds__(kThreads) k_na_setup(SysDev S, NaPtrs p) {
  const long long K = static_cast<long long>(S.grid[0]) * S.grid[1] * S.grid[2];
  for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += gridDim.x * blockDim.x) p.grid[i] = 0ull;
  __shared__ double co[kNoAllocMaxAxis], si[kNoAllocMaxAxis];
  __shared__ float mod[kNoAllocMaxAxis];
  for (int axis = blockIdx.x; axis < 3; axis += gridDim.x) {
    const int n = S.grid[axis];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      sincospi(2.0 * j / n, &si[j], &co[j]);
      p.twiddles[axis * kNoAllocMaxAxis + j] = make_float2(float(co[j]), float(-si[j]));
    }
    __syncthreads();
    const double knots[4] = {1.0 / 24, 11.0 / 24, 11.0 / 24, 1.0 / 24};
    for (int m = threadIdx.x; m < n; m += blockDim.x) {
      double re = 0, im = 0;
      for (int k = 0; k < 4; ++k) {  // an axis has at least five points
        re += knots[k] * co[(m * k) % n];
        im += knots[k] * si[(m * k) % n];
      }
      mod[m] = float(re * re + im * im);
    }
    __syncthreads();
    // bspline.ts:126 -- replace a vanishing modulus by its neighbours' mean.
    // Of an order-5 spline's only the one at n/2 of an even axis vanishes, so
    // no neighbour is itself one to be replaced.
    for (int m = threadIdx.x; m < n; m += blockDim.x) {
      float* out = p.moduli + axis * kNoAllocMaxAxis;
      const float before = mod[(m - 1 + n) % n], after = mod[(m + 1) % n];
      out[m] = mod[m] < 1e-7f ? 0.5f * (before + after) : mod[m];
    }
    __syncthreads();
  }
}

__device__ __forceinline__ long long fixed_from_double(double x) { return __double2ll_rn(x * 4294967296.0); }

// By atom: the caller's order says nothing about where the atoms are.  A
// block computes its atoms' splines once (a thread per atom and axis), then
// shares the 25 rows of 5 z points per atom over its threads.
constexpr int kNaAtoms = 32;

__global__ void __launch_bounds__(kThreads) k_na_spread(SysDev S, NaPtrs p, int n, const double* pos,
                                                        const double* charge) {
  wait_for_predecessor();
  __shared__ int base[kNaAtoms][3];
  __shared__ float th[kNaAtoms][3][5], qs[kNaAtoms];
  const int first = blockIdx.x * kNaAtoms;
  for (int w = threadIdx.x; w < 3 * kNaAtoms; w += blockDim.x) {
    const int axis = w / kNaAtoms, k = w - axis * kNaAtoms, i = first + k;
    const float q = i < n ? float(charge[i]) : 0.f;
    if (axis == 0) qs[k] = q;
    if (q == 0.f) continue;
    float weights[5];
    base[k][axis] = spline_axis(S, axis, fixed_from_double(pos[3 * i]), fixed_from_double(pos[3 * i + 1]),
                                fixed_from_double(pos[3 * i + 2]), weights, nullptr);
#pragma unroll
    for (int j = 0; j < kPmeOrder; ++j) th[k][axis][j] = weights[j];
  }
  __syncthreads();
  const int Kx = S.grid[0], Ky = S.grid[1], Kz = S.grid[2];
  for (int w = threadIdx.x; w < kNaAtoms * kPmeOrder * kPmeOrder; w += blockDim.x) {
    const int k = w / (kPmeOrder * kPmeOrder), r = w - k * kPmeOrder * kPmeOrder;
    const float q = qs[k];
    if (q == 0.f) continue;
    const int ix = r / kPmeOrder, iy = r - ix * kPmeOrder;
    int gx = base[k][0] + ix, gy = base[k][1] + iy;
    if (gx >= Kx) gx -= Kx;
    if (gy >= Ky) gy -= Ky;
    const float wxy = q * th[k][0][ix] * th[k][1][iy];
    unsigned long long* row = p.grid + (static_cast<long long>(gx) * Ky + gy) * Kz;
#pragma unroll
    for (int iz = 0; iz < kPmeOrder; ++iz) {
      int gz = base[k][2] + iz;
      if (gz >= Kz) gz -= Kz;
      add_fixed(&row[gz], wxy * th[k][2][iz]);
    }
  }
}

__device__ __forceinline__ Mesh mesh_of(const SysDev& S, const NaPtrs& p) {
  Mesh m;
  m.x = {S.grid[0], S.plan[0]};
  m.y = {S.grid[1], S.plan[1]};
  m.z = {S.grid[2], S.plan[2]};
  m.kzh = S.kzh;
  m.charge = p.grid;
  m.spectrum = p.spectrum;
  m.potential = p.potential;
  m.twx = p.twiddles;
  m.twy = p.twiddles + kNoAllocMaxAxis;
  m.twz = p.twiddles + 2 * kNoAllocMaxAxis;
  return m;
}

// The engine's passes over this mesh: block b of each takes plane b, or strip
// b of a plane.
__global__ void __launch_bounds__(kPlaneThreads) k_na_planes_forward(SysDev S, NaPtrs p) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  plane_forward(mesh_of(S, p), blockIdx.x, smem);
}
__global__ void __launch_bounds__(kPlaneThreads) k_na_planes_inverse(SysDev S, NaPtrs p) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  plane_inverse(mesh_of(S, p), blockIdx.x, smem);
}
// z and y passes for planes that do not fit shared memory: `lines` (even) z
// lines of a plane, kFftTile columns of one
__global__ void __launch_bounds__(kThreads) k_na_z_forward(SysDev S, NaPtrs p, int lines) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const int Ky = S.grid[1], per = (Ky + lines - 1) / lines, x = blockIdx.x / per, y = (blockIdx.x - x * per) * lines;
  z_forward(mesh_of(S, p), x * Ky + y, min(lines, Ky - y), smem);
}
__global__ void __launch_bounds__(kThreads) k_na_z_inverse(SysDev S, NaPtrs p, int lines) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const int Ky = S.grid[1], per = (Ky + lines - 1) / lines, x = blockIdx.x / per, y = (blockIdx.x - x * per) * lines;
  z_inverse(mesh_of(S, p), x * Ky + y, min(lines, Ky - y), smem);
}
template <int SIGN>
__global__ void __launch_bounds__(kThreads) k_na_y(SysDev S, NaPtrs p) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const int per = (S.kzh + kFftTile - 1) / kFftTile, x = blockIdx.x / per, kz0 = (blockIdx.x - x * per) * kFftTile;
  y_pass<SIGN>(mesh_of(S, p), x, kz0, min(kFftTile, S.kzh - kz0), smem);
}

__global__ void __launch_bounds__(kXThreads) k_na_x_convolve(SysDev S, NaPtrs p) {
  wait_for_predecessor();
  extern __shared__ float2 smem[];
  const int per = (S.kzh + kFftTile - 1) / kFftTile, my = blockIdx.x / per, kz0 = (blockIdx.x - my * per) * kFftTile;
  const int Kx = S.grid[0], Ky = S.grid[1], Kz = S.grid[2], mb = my <= Ky / 2 ? my : my - Ky;
  double energy[1] = {0.0};
  x_pass(mesh_of(S, p), my, kz0, min(kFftTile, S.kzh - kz0), smem, [&](int mx, int l, float2 v) {
    const int kz = kz0 + l;
    float kx, ky, kzv, k2;
    const float f = influence(S, p.moduli, p.moduli + kNoAllocMaxAxis, p.moduli + 2 * kNoAllocMaxAxis, Kx, mx, mb, my, kz,
                              kx, ky, kzv, k2);
    const double weight = (kz == 0 || (2 * kz == Kz)) ? 1.0 : 2.0;
    energy[0] += weight * double(f) * (double(v.x) * v.x + double(v.y) * v.y);
    const float g = 2.f * f;
    return make_float2(__fmul_rn(v.x, g), __fmul_rn(v.y, g));
  });
  block_sums<1>(energy, [&](int, double total) { p.partials[blockIdx.x] = total; });
}

// Forces; and, by the last block's first warp, the energy from the x pass'
// `count` partial sums, in a fixed order.
__global__ void __launch_bounds__(kGatherThreads) k_na_gather(SysDev S, NaPtrs p, int n, const double* pos,
                                                              const double* charge, double* forces, int count,
                                                              double* energy) {
  wait_for_predecessor();
  __shared__ GatherTable table;
  if (blockIdx.x == gridDim.x - 1) {  // the whole block
    if (threadIdx.x < 32) {
      double total = 0.0;
      for (int k = threadIdx.x; k < count; k += 32) total += p.partials[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
      if (threadIdx.x == 0) *energy = total;
    }
    return;
  }
  const int i = blockIdx.x * kGatherAtoms + (threadIdx.x & 31);
  const float q = i < n ? float(charge[i]) : 0.f;
  const bool live = q != 0.f;
  if (i < n && !live && threadIdx.x < 32) forces[3 * i] = forces[3 * i + 1] = forces[3 * i + 2] = 0.0;
  float ga, gb, gc;
  if (!gather_block(table, live, S, p.potential, live ? fixed_from_double(pos[3 * i]) : 0,
                    live ? fixed_from_double(pos[3 * i + 1]) : 0, live ? fixed_from_double(pos[3 * i + 2]) : 0, ga, gb,
                    gc))
    return;
  const float3 f = mesh_force(S, q, ga, gb, gc);
  forces[3 * i] = f.x;
  forces[3 * i + 1] = f.y;
  forces[3 * i + 2] = f.z;
}

// The scratch array's device address, looked up with the device current.  In
// host code `g_noalloc_scratch` names a host-side stand-in, never device
// memory, so kernels must be given this address instead.  A call on a stream
// that is not capturing looks the address up again (cheap), so a device reset,
// which reloads the module at a new address, is picked up by the next such
// call; a call inside a stream capture uses the address the last call outside
// one found, and fails if there is none yet.
std::mutex g_noalloc_mutex;
std::array<unsigned char*, 64> g_noalloc_address{};

int noalloc_scratch(int device, bool capturing, unsigned char** out) {
  if (device < 0 || device >= int(g_noalloc_address.size())) return MDB_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!capturing) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || ptr == nullptr) return MDB_ERR_DEVICE;
    g_noalloc_address[device] = static_cast<unsigned char*>(ptr);
  }
  if (!g_noalloc_address[device]) return MDB_ERR_INVALID_ARGUMENT;
  *out = g_noalloc_address[device];
  return MDB_OK;
}

}  // namespace
}  // namespace mdb

extern "C" int mdb_reciprocal_noalloc(int32_t n, const double* positions, const double* charges,
                                      const double box[9], double alpha, const int32_t mesh[3], double* forces,
                                      double* energy, void* stream) {
  using namespace mdb;
  if (n < 0 || !box || !mesh || !energy || !(alpha > 0) || (n > 0 && (!positions || !charges || !forces)))
    return MDB_ERR_INVALID_ARGUMENT;
  long long points = 1;
  for (int k = 0; k < 3; ++k) {
    // an order-5 spline spans 5 mesh points, wrapped once into the mesh
    if (mesh[k] < kPmeOrder) return MDB_ERR_INVALID_ARGUMENT;
    if (mesh[k] > kNoAllocMaxAxis) return MDB_ERR_CAPACITY;
    points *= mesh[k];
  }
  if (points > kNoAllocMaxMeshPoints) return MDB_ERR_CAPACITY;
  SysDev S;
  std::memset(&S, 0, sizeof(S));
  for (int k = 0; k < 3; ++k) {
    S.grid[k] = mesh[k];
    if (!plan_radices(mesh[k], &S.plan[k])) return MDB_ERR_NOT_SMOOTH;
  }
  S.kzh = mesh[2] / 2 + 1;
  double B[9], M[9];
  if (!reduce_box(box, B)) return MDB_ERR_INVALID_ARGUMENT;
  inverse_box(B, M);
  for (int i = 0; i < 9; ++i) S.inv_f[i] = float(M[i]);
  const double um[6] = {mesh[0] * M[0], mesh[0] * M[3], mesh[0] * M[6], mesh[1] * M[4], mesh[1] * M[7], mesh[2] * M[8]};
  for (int i = 0; i < 6; ++i) S.umat[i] = std::llround(um[i] * 4294967296.0);
  for (int v = 0; v < 3; ++v)
    for (int u = 0; u < 3; ++u) S.umat_f[v * 3 + u] = float(mesh[u] * M[v * 3 + u]);
  S.pme_pref = float(kOne4PiEps0 * 2 * 3.14159265358979323846 / box_volume(B));
  S.exp_scale = float(-1.0 / (4 * alpha * alpha));

  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return MDB_ERR_NO_DEVICE;
  // An error left by the caller's earlier work is theirs: report it without
  // consuming it, so that only this call's own launches set what
  // cudaGetLastError returns below.
  if (cudaPeekAtLastError() != cudaSuccess) return MDB_ERR_DEVICE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) return MDB_ERR_DEVICE;
  unsigned char* base = nullptr;
  const int status = noalloc_scratch(device, capture != cudaStreamCaptureStatusNone, &base);
  if (status != MDB_OK) return status;
  NaPtrs p;
  p.grid = reinterpret_cast<unsigned long long*>(base + kNaGrid);
  p.spectrum = reinterpret_cast<float2*>(base + kNaSpectrum);
  p.potential = reinterpret_cast<float*>(base + kNaPotential);
  p.moduli = reinterpret_cast<float*>(base + kNaModuli);
  p.twiddles = reinterpret_cast<float2*>(base + kNaTwiddles);
  p.partials = reinterpret_cast<double*>(base + kNaPartials);

  const int Kx = mesh[0], Ky = mesh[1], Kz = mesh[2];
  const int tiles = (S.kzh + kFftTile - 1) / kFftTile;
  k_na_setup<<<std::max(3, int(std::min<long long>((points + 1023) / 1024, 148 * 4))), kThreads, 0, st>>>(S, p);
  if (n > 0) launch_chained(k_na_spread, (n + kNaAtoms - 1) / kNaAtoms, kThreads, 0, st, S, p, n, positions, charges);
  const int plane = plane_smem(Ky, Kz), lines = std::max(2, 2048 / Kz & ~1);
  if (plane <= kNoAllocPlaneSmem) {
    launch_chained(k_na_planes_forward, Kx, kPlaneThreads, plane, st, S, p);
  } else {
    launch_chained(k_na_z_forward, Kx * ((Ky + lines - 1) / lines), kThreads, z_smem(lines, Kz), st, S, p, lines);
    launch_chained(k_na_y<-1>, Kx * tiles, kThreads, strip_smem(kFftTile, Ky), st, S, p);
  }
  launch_chained(k_na_x_convolve, Ky * tiles, kXThreads, strip_smem(kFftTile, Kx), st, S, p);
  if (plane <= kNoAllocPlaneSmem) {
    launch_chained(k_na_planes_inverse, Kx, kPlaneThreads, plane, st, S, p);
  } else {
    launch_chained(k_na_y<+1>, Kx * tiles, kThreads, strip_smem(kFftTile, Ky), st, S, p);
    launch_chained(k_na_z_inverse, Kx * ((Ky + lines - 1) / lines), kThreads, z_smem(lines, Kz), st, S, p, lines);
  }
  launch_chained(k_na_gather, (n + kGatherAtoms - 1) / kGatherAtoms + 1, kGatherThreads, 0, st, S, p, n, positions, charges,
                 forces, Ky * tiles, energy);
  return cudaGetLastError() == cudaSuccess ? MDB_OK : MDB_ERR_DEVICE;
}
