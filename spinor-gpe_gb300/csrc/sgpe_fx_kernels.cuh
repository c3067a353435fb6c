// Pass kernels of the complex128 precision in 64-bit fixed point
// (sgpe_fx.cuh).  The state stays FP64 in memory; a block turns its lines
// into integers with one exponent per line, runs transforms, operators and
// sums on them, and writes FP64 again.  Same passes, arguments and tiles as
// col_body / row_body.
//
// Bound: integer issue.  At 1024^2 a column pass issues 511 instructions per
// point and component (wide multiply-adds take their pipe for 2-2.6 cycles)
// and a row pass 760, at two instructions per cycle and SM; DRAM and L2 are
// under 15% busy.  Measured at 1024^2 (real time, Raman coupling; column / row
// / step): FP64 butterflies 347 / 473 / 2,470 us, fixed point 60.7 / 84.1 /
// 403 us, with half the error against the same operations in 80 bits (90
// problems of 2 to 20 steps, 32 x 512 to 4096 x 32: geometric mean 0.47 of the
// FP64 kernels').
#pragma once
#include "sgpe_kernels.cuh"

namespace sgpe {

// Scaling 2^-q of a transform of (N, E): of every stage after the first, or
// (LAST false) of those in front of the last.
template <int N, int E, bool LAST = true> __host__ __device__ constexpr int fx_transform_q() {
  int q = 0, ns = stage_radix(N, E, 1);
  while (ns < N) {
    const int r = stage_radix(N, E, ns);
    if (LAST || ns * r < N) q += fx_bits(r);
    ns *= r;
  }
  return q;
}

// A thread's share of its line's L1 norm in units of 2^44, rounded up: the
// high words' magnitudes fit 32 bits for |z| < 2^(62.5 - bits(E)).
template <int E> __device__ __forceinline__ uint32_t fx_l1(const FxC (&v)[E]) {
  uint32_t s = 2 * E;
#pragma unroll
  for (int m = 0; m < E; ++m)
    s += uint32_t(abs(int(v[m].x >> 32))) + uint32_t(abs(int(v[m].y >> 32)));
  return (s >> 12) + 1;
}

// Largest magnitude of a thread's parts (high words), and the shift that
// brings a line with that largest value up to the headroom of its first stage.
template <int E> __device__ __forceinline__ uint32_t fx_max(const FxC (&v)[E]) {
  uint32_t s = 0;
#pragma unroll
  for (int m = 0; m < E; ++m)
    s = max(s, max(uint32_t(abs(int(v[m].x >> 32))), uint32_t(abs(int(v[m].y >> 32)))));
  return s;
}
__device__ __forceinline__ int fx_pre(uint32_t largest, int bits) {
  return max(0, min(__clz(int(largest + 1)) - 2 - bits, 24));
}

// Components that a coupling mixes are held at one exponent where theirs are
// at most this far apart (of 59 bits two go), and at their own where they are
// further: a polarised gas under a weak drive keeps the bits of its minority
// (two steps from 1e-6 of the other's amplitude at omega = 1e-3: 7e-11 of
// itself with one exponent, 4e-16 so).
constexpr int kFxUnlike = 2;

// The exchange lines of a fixed-point transform.  A line's L1 norm is what
// its threads know (own) plus `warps` entries in shared memory, written in
// front of the transform's first exchange.  PAIR: the norm of the row's other
// component too; lines loaded with one exponent (common) shift alike, unless
// one of them has much more room than the other.
template <int N, int E, bool WARP, bool PAIR> struct FxLine : LineSmem<FxC, E, WARP> {
  const uint32_t* l1;
  const uint32_t* l1_other;
  int warps, stride;
  uint32_t own, own_other;
  bool common;
  int pre = 0;   // shift of the line in front of its first stage (part of `shift`)
  mutable int shift = 0, shift_other = 0;
  __device__ __forceinline__ FxLine(FxC* base, int warps_, int stride_, const uint32_t* l1_, uint32_t own_ = 0,
                                    const uint32_t* l1o = nullptr, uint32_t owno = 0, bool common_ = false)
      : LineSmem<FxC, E, WARP>{base, 0}, l1(l1_), l1_other(l1o), warps(warps_), stride(stride_), own(own_),
        own_other(owno), common(common_) {}
  __device__ __forceinline__ int up() const {
    uint32_t s = own, t = own_other;
#pragma unroll
    for (int w = 0; w < warps; ++w) {
      s += l1[w * stride];
      if (PAIR) t += l1_other[w * stride];
    }
    constexpr int kScaled = fx_transform_q<N, E, false>();
    int u = fx_room(s, kScaled - pre);
    if (PAIR) {
      shift_other = fx_room(t, kScaled);
      if (common && abs(u - shift_other) <= kFxUnlike) u = shift_other = min(u, shift_other);
    }
    shift = u + pre;
    return u;
  }
};

__device__ __forceinline__ uint32_t fx_hi_max(uint32_t m, int4 w) {
  const uint32_t a = uint32_t(w.y) & 0x7fffffffu, b = uint32_t(w.w) & 0x7fffffffu;
  return max(m, max(a, b));
}
// FP64 <-> integer through the conversion instructions: at 48 cycles of the
// otherwise idle FP64 pipe they leave the integer pipes, which bound these
// kernels, 7 instructions a value instead of 39 (sgpe_fx.cuh's word forms).
// The power of two goes into the exponent field.  Where the pipe would be
// waited for, the word forms stay: with 12 points per thread (sides 3 * 2^k:
// a 768^2 transform pair 98 against 108 us), in the small shapes of 4,
// with a few warps per SM, and on lines of 4096, whose one block per SM
// converts all at once (us a step, instructions / words: 1024^2 411 / 422;
// 2048^2 1,754 / 1,778; 256^2 56.4 / 53.3, 4096^2 8,300 / 7,858).
__host__ __device__ constexpr bool fx_convert(int n, int e) { return e == 8 && n <= 2048; }
__device__ __forceinline__ fx_t fx_load_part(uint32_t hi, uint32_t lo, int q) {
  const int e = q << 20;
  // below the normal range after the scaling: reads as zero (2^-62 of the line)
  const bool tiny = int(hi & 0x7fffffffu) - e < 0x100000;
  return __double2ll_rn(__hiloint2double(tiny ? 0 : int(hi) - e, int(lo)));
}
// a value of a line of biased exponent be at |part| < 2^p
template <bool CONVERT> __device__ __forceinline__ FxC fx_load(int4 w, int be, int p) {
  if constexpr (CONVERT) {
    const int q = fx_line_q(be, p);
    return FxC{fx_load_part(uint32_t(w.y), uint32_t(w.x), q), fx_load_part(uint32_t(w.w), uint32_t(w.z), q)};
  } else {
    return FxC{fx_from_words(uint32_t(w.y), uint32_t(w.x), be, p), fx_from_words(uint32_t(w.w), uint32_t(w.z), be, p)};
  }
}
// v 2^q for any q (overflow to infinity, underflow to zero)
static __device__ __noinline__ double fx_to_double_far(fx_t v, int q) {
  return ldexp(ldexp(double(v), q / 2), q - q / 2);
}
// ... for q in the range of fx_q_safe
__device__ __forceinline__ double fx_to_double_near(fx_t v, int q) {
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d);
  return __hiloint2double(v == 0 ? 0 : hi + (q << 20), __double2loint(d));
}
__device__ __forceinline__ double fx_to_double(fx_t v, int q) {
  return fx_q_safe(q) ? fx_to_double_near(v, q) : fx_to_double_far(v, q);
}
// What a line's element is written as: v 2^q, or NaN in a bad line.
enum FxOut { kFxNear = 0, kFxFar = 1, kFxBad = 2 };
__device__ __forceinline__ FxOut fx_out(bool bad, int q) { return bad ? kFxBad : fx_q_safe(q) ? kFxNear : kFxFar; }
template <FxOut OUT, bool CONVERT> __device__ __forceinline__ int4 fx_words(FxC v, int q) {
  if constexpr (OUT == kFxBad) return make_int4(0, 0x7ff80000, 0, 0x7ff80000);
  if constexpr (OUT == kFxNear && !CONVERT) {
    uint32_t xh, xl, yh, yl;
    fx_to_words(v.x, q, &xh, &xl);
    fx_to_words(v.y, q, &yh, &yl);
    return make_int4(int(xl), int(xh), int(yl), int(yh));
  }
  const double x = OUT == kFxNear ? fx_to_double_near(v.x, q) : fx_to_double_far(v.x, q);
  const double y = OUT == kFxNear ? fx_to_double_near(v.y, q) : fx_to_double_far(v.y, q);
  return make_int4(__double2loint(x), __double2hiint(x), __double2loint(y), __double2hiint(y));
}
constexpr int kNanHi = 0x7ff80000;

// A real factor as a mantissa |m| < 2^62 and its exponent.
struct FxScale {
  FxSplit m;
  int e;
  bool finite;
};
__device__ __forceinline__ FxScale fx_scale(double s) {
  const uint32_t hi = uint32_t(__double2hiint(s)), lo = uint32_t(__double2loint(s));
  const int be = fx_line_exp(hi & 0x7fffffffu);
  return FxScale{fx_split(fx_from_words(hi, lo, be, 62)), fx_line_q(be, 62), be != kFxNonFinite};
}

// Sum of |v|^2 over a thread's E points, |v|^2 summing below 2^121, in units
// of 2^43 as three limbs of 26 bits (the upper one of up to 27): rounding far
// below anything a line's norm can see, and 32 lanes' limbs add up in 32 bits.
struct FxSum {
  uint32_t low, mid, top;
};
template <int E> __device__ __forceinline__ FxSum fx_norm2(const FxC (&v)[E]) {
  fx_t hh = 0, hl = 0, ll = 0;  // squares of the high words, cross terms, low words in 2^16 steps
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const FxSplit x = fx_split(v[m].x), y = fx_split(v[m].y);
    hh = fx_mad(x.h, x.h, fx_mad(y.h, y.h, hh));
    hl = fx_mad(x.h, x.l, fx_mad(y.h, y.l, hl));
    ll = fx_mad(x.l >> 8, x.l >> 8, fx_mad(y.l >> 8, y.l >> 8, ll));
  }
  // hh 2^64 + hl 2^33 + ll 2^16
  const fx_t a = (hl >> 10) + (ll >> 27) + ((hh & 31) << 21);
  const fx_t m = (a >> 26) + (hh >> 5);
  constexpr uint32_t kMask = (1u << 26) - 1;
  return FxSum{uint32_t(a) & kMask, uint32_t(m) & kMask, uint32_t(m >> 26)};
}
// The sum over a warp's lanes of one column.
template <int COLS> __device__ __forceinline__ FxSum fx_column_sum(FxSum s) {
#pragma unroll
  for (int o = 16; o >= COLS; o >>= 1) {
    s.low += __shfl_xor_sync(0xffffffffu, s.low, o);
    s.mid += __shfl_xor_sync(0xffffffffu, s.mid, o);
    s.top += __shfl_xor_sync(0xffffffffu, s.top, o);
  }
  return s;
}
// The sum of N such sums, STRIDE apart, times 2^q.
template <int N, int STRIDE> __device__ __forceinline__ double fx_sum_value(const FxSum* s, int q) {
  uint64_t low = 0, mid = 0, top = 0;
  for (int i = 0; i < N; ++i) {
    low += s[i * STRIDE].low;
    mid += s[i * STRIDE].mid;
    top += s[i * STRIDE].top;
  }
  return fx_to_double(fx_t((top << 26) + mid), q + 69) + fx_to_double(fx_t(low), q + 43);
}

// v[m] *= ka(x) kb(ky) 2^-2 along a column; returns what the exponent gains.
// The column's factor ka keeps its own exponent (it is tiny for the high
// momenta of an imaginary-time step).
template <int E, int T>
__device__ __forceinline__ int fx_kinetic(FxC (&v)[E], const double2* __restrict__ ka, const int4* __restrict__ kb,
                                          int eb, int x, int j) {
  const int4 w = __ldg(reinterpret_cast<const int4*>(ka) + x);
  const int be = fx_line_exp(fx_hi_max(0, w));
  const FxC a = fx_load<false>(w, be, 61);
  const FxSplit ax = fx_split(a.x), ay = fx_split(a.y);
#pragma unroll
  for (int m = 0; m < E; ++m) {
    // |ka| < 2^61.5, kb up to 2^62: the product up to 2^59.5, times 2^2
    const FxC k = fx_cmul<false>(ax, ay, __ldg(kb + j + m * T), FxC{0, 0});
    v[m] = fx_cmul<false>(v[m], fx_factor(k.x << 2, k.y << 2));
  }
  return eb + fx_line_q(be, 61) + 64;
}

// -------------------------------------------------------------- column pass
// largest of a column's entries in shared memory, one per warp
template <int NW, int COLS> __device__ __forceinline__ uint32_t fx_max_entries(const uint32_t* s, int lane) {
  uint32_t mx = 0;
#pragma unroll
  for (int i = 0; i < (NW * COLS + 31) / 32; ++i)
    if (lane + 32 * i < NW * COLS) mx = max(mx, s[lane + 32 * i]);
#pragma unroll
  for (int o = 16; o >= COLS; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

template <int N, int E, int COLS>
__device__ __forceinline__ void col_body_fx(const ColArgs<double>& a, const BlockPos pos) {
  constexpr int T = N / E;
  constexpr int LS = column_line_stride(N, E, COLS, sizeof(FxC));
  constexpr int NT = T * COLS;
  constexpr int NW = NT / 32;
  constexpr int kBits = fx_bits(stage_radix(N, E, 1));
  constexpr int kTq = fx_transform_q<N, E>();
  static_assert(COLS <= 32 && (COLS & (COLS - 1)) == 0 && NT % 32 == 0, "whole warps of whole column groups");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FxC* sm = reinterpret_cast<FxC*>(smem_raw);
  __shared__ uint32_t s_mx[NW * COLS], s_mx2[NW * COLS];
  __shared__ uint32_t s_l1[2][NW * COLS];
  __shared__ FxSum s_sum[2][NW * COLS];
  __shared__ double s_line[2][COLS];

  const int tid = threadIdx.x;
  const int c = tid % COLS;
  const int j = tid / COLS;
  const int warp = tid >> 5, lane = tid & 31;
  const int comp = pos.y;
  const int nx = a.nx;
  const int x = pos.x * COLS + c;
  const int half = nx / 2;
  const int xin = a.in_shift ? (x + half) % nx : x;
  const int xout = a.out_shift ? (x + half) % nx : x;
  const int4* __restrict__ in = reinterpret_cast<const int4*>(a.in[comp]);
  int4* out = reinterpret_cast<int4*>(a.out[comp]);

  FxC v[1][E];
  int q;
  bool bad;
  {
    int4 w[E];
    wait_for_previous_grid();
    {
      // rows j + m T; in centred order the two halves change places
      const long long step = (long long)T * nx, swap = a.in_shift ? E / 2 * step : 0;
      const int4* p = in + (long long)j * nx + xin + swap;
#pragma unroll
      for (int m = 0; m < E; ++m, p += step) {
        if (m == E / 2) p -= 2 * swap;
        w[m] = *p;
      }
    }
    allow_next_grid();
    // largest exponent of the column: over its lanes, then over the warps
    uint32_t mx = 0;
#pragma unroll
    for (int m = 0; m < E; ++m) mx = fx_hi_max(mx, w[m]);
#pragma unroll
    for (int o = 16; o >= COLS; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if constexpr (NW > 1) {
      if (lane < COLS) s_mx[warp * COLS + lane] = mx;
      __syncthreads();
      mx = fx_max_entries<NW, COLS>(s_mx, lane);
    }
    const int be = fx_line_exp(mx);
    bad = be == kFxNonFinite;
    // a line that meets a kinetic factor (2^-2) before its transform needs
    // less headroom for the first stage
    const int p = (!a.fwd && a.nk > 0) ? 63 - kBits : 62 - kBits;
    q = fx_line_q(be, p);
#pragma unroll
    for (int m = 0; m < E; ++m) v[0][m] = fx_load<fx_convert(N, E)>(w[m], be, p);
  }
  const FxC* tw = reinterpret_cast<const FxC*>(a.twf);
  using Line = FxLine<N, E, false, false>;
  auto line_l1 = [&](int k) {
    uint32_t s = fx_l1<E>(v[0]);
#pragma unroll
    for (int o = 16; o >= COLS; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < COLS) s_l1[k][warp * COLS + lane] = s;
    return Line(sm + c * LS, NW, COLS, s_l1[k] + c);
  };
  if (a.fwd) {
    const auto smv = line_l1(0);
    fft_lines<N, E, -1, 1>(v, j, smv, tw);
    q += kTq - smv.shift;
  }
  // populations u and norm w of the column, summed as integers
  FxSum su{0, 0, 0}, sw{0, 0, 0};
  int qu = 0;
  if (a.nk > 0) {
    q += fx_kinetic<E, T>(v[0], a.k1.a[comp].p, a.kb[0][comp], a.ke[0][comp], x, j);
    if (a.nk == 2) {
      su = fx_norm2<E>(v[0]);
      qu = q;
      q += fx_kinetic<E, T>(v[0], a.k2.a[comp].p, a.kb[1][comp], a.ke[1][comp], x, j);
    }
    if (a.part != nullptr) sw = fx_norm2<E>(v[0]);
  }
  const int qw = q;
  if (a.inv) {
    Line smv = line_l1(1);
    if (a.nk > 0) {
      // what the factors took and what the spectrum left free goes back
      // in front of the transform
      uint32_t mx = fx_max<E>(v[0]);
#pragma unroll
      for (int o = 16; o >= COLS; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane < COLS) s_mx2[warp * COLS + lane] = mx;
      __syncthreads();
      mx = fx_max_entries<NW, COLS>(s_mx2, lane);
      smv.pre = fx_pre(mx, kBits);
#pragma unroll
      for (int m = 0; m < E; ++m) v[0][m] = FxC{v[0][m].x << smv.pre, v[0][m].y << smv.pre};
    }
    fft_lines<N, E, +1, 1>(v, j, smv, tw);
    q += kTq - smv.shift;
  }
  int qo = q;
  if (a.scale != 1.0) {
    const FxScale s = fx_scale(a.scale);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      v[0][m].x = fx_mul(fx_split(v[0][m].x), s.m);
      v[0][m].y = fx_mul(fx_split(v[0][m].y), s.m);
    }
    qo += 64 + s.e;
    bad = bad || !s.finite;
  }
  {
    const long long step = (long long)T * nx, swap = a.out_shift ? E / 2 * step : 0;
    int4* const first = out + (long long)j * nx + xout + swap;
    auto write = [&](auto form) {
      int4* p = first;
#pragma unroll
      for (int m = 0; m < E; ++m, p += step) {
        if (m == E / 2) p -= 2 * swap;
        *p = fx_words<decltype(form)::value, fx_convert(N, E)>(v[0][m], qo);
      }
    };
    const FxOut form = fx_out(bad, qo);
    if (form == kFxNear) write(std::integral_constant<FxOut, kFxNear>{});
    else if (form == kFxBad) write(std::integral_constant<FxOut, kFxBad>{});
    else write(std::integral_constant<FxOut, kFxFar>{});
  }
  if (a.part != nullptr) {
    sw = fx_column_sum<COLS>(sw);
    if (a.nk == 2) su = fx_column_sum<COLS>(su);
    if (lane < COLS) {
      s_sum[0][warp * COLS + lane] = su;
      s_sum[1][warp * COLS + lane] = sw;
    }
    __syncthreads();
    if (tid < COLS) {
      const double lw = fx_sum_value<NW, COLS>(&s_sum[1][tid], 2 * qw);
      const double lu = a.nk == 2 ? fx_sum_value<NW, COLS>(&s_sum[0][tid], 2 * qu) : lw;
      const double nan = __hiloint2double(kNanHi, 0);
      s_line[0][tid] = bad ? nan : lu;
      s_line[1][tid] = bad ? nan : lw;
    }
    if constexpr (COLS > 1) __syncwarp();
    if (tid == 0) {
      double bu = 0.0, bw = 0.0;
#pragma unroll
      for (int k = 0; k < COLS; ++k) {
        bu += s_line[0][k];
        bw += s_line[1][k];
      }
      double* dst = a.part + 2 * ((long long)comp * pos.nx + pos.x);
      dst[0] = bu;
      dst[1] = bw;
    }
    col_finish(a, pos, tid, NT);
  }
}

template <int N, int E, int COLS, int MINB>
__global__ void __launch_bounds__((N / E) * COLS, MINB)
col_kernel_fx(const ColArgs<double> a) {
  col_body_fx<N, E, COLS>(a, grid_pos());
}
template <int N, int E, int COLS, int MINB>
__global__ void __launch_bounds__((N / E) * COLS, MINB)
col_kernel_fx_grouped(const ColArgs<double>* __restrict__ args) {
  col_body_fx<N, E, COLS>(args[blockIdx.z], grid_pos());
}

// ----------------------------------------------------------------- row pass
// Exact sums of non-negative FP64 values (the column pass's partials) over a
// block: each value in 72 bits below the largest one's exponent, three limbs
// of 24 bits whose sums over a warp (up to four values a thread) fit 32 bits.
struct FxLimbs {
  uint32_t l[3];
};
__device__ __forceinline__ void fx_limb_add(FxLimbs* s, double v, int be) {
  const uint32_t hi = uint32_t(__double2hiint(v)), lo = uint32_t(__double2loint(v));
  const uint32_t e = hi >> 20;
  const uint64_t m = (uint64_t((hi << 11) | (lo >> 21) | (e ? 0x80000000u : 0u)) << 32) | (lo << 11);
  const int d = be - int(e ? e : 1);       // below the largest exponent (subnormals and zeros: exponent 1)
  const uint64_t t = fx_shr(m, d);         // the upper 64 bits
  const uint64_t r = d == 0 ? 0 : d < 64 ? m << (64 - d) : fx_shr(m, d - 64);
  s->l[0] += uint32_t(t >> 40);
  s->l[1] += uint32_t(t >> 16) & 0xffffffu;
  s->l[2] += (uint32_t(t & 0xffffu) << 8) | uint32_t(r >> 56);
}
// sum of the warps' limbs, times 2^q of one in the last of the 72 bits
__device__ __forceinline__ double fx_limb_value(const FxLimbs* s, int warps, int be) {
  uint64_t a = 0, b = 0, c = 0;
  for (int w = 0; w < warps; ++w) {
    a += s[w].l[0];
    b += s[w].l[1];
    c += s[w].l[2];
  }
  // the largest exponent's values lie in [2^71, 2^72) units
  const int q = be - 1023 - 71;
  return fx_to_double(fx_t((a << 24) + b), q + 24) + fx_to_double(fx_t(c), q);
}

// The populations from the column pass's partial sums [comp][tile][u, w] (or
// their final sums), summed in FP64 by one warp of block 0 while the others wait
// for the row's constants.  (A call, as above.)
static __device__ __noinline__ void fx_populations(const double* part, const double* fin, int ntile, double atom_num,
                                                   double* pops) {
  const int lane = threadIdx.x & 31;
  double u0 = 0.0, u1 = 0.0;
  if (fin == nullptr) {
    for (int i = lane; i < ntile; i += 32) {
      u0 += part[2 * i];
      u1 += part[2 * (ntile + i)];
    }
    u0 = warp_sum(u0);
    u1 = warp_sum(u1);
  } else {
    u0 = fin[0];
    u1 = fin[1];
  }
  if (lane == 0) {
    pops[0] = atom_num * u0 / (u0 + u1);
    pops[1] = atom_num * u1 / (u0 + u1);
  }
}

// What the point-wise operators of one row share.
struct FxRow {
  int4 pb;           // pb(y) lambda
  FxSplit m[2][2];   // phase of component i per |z_j|^2 (times 2^-twice)
  int sh[2];         // |z_j|^2 is shifted left by this before the product
  int twice;         // the phases come out times 2^-twice
  int qm[2];         // exponent of the components behind the matrix
  int q[2];          // ... and of their lines in front of F_x
  int dm[4];         // with the matrix of own exponents: shift of each product
  bool split;        // take that one
  bool bad;
};

// e^{i 2^twice x} - 1 as a split factor, x = X 2^-64, the phase at most 1/2
__device__ __forceinline__ int4 fx_phase(fx_t X, int twice) {
  fx_t sn, cm;
  fx_sincos(X, &sn, &cm);
  for (int k = 0; k < twice; ++k) {  // sin 2x = 2 (sin x + sin x (cos x - 1)), cos 2x - 1 = -2 sin^2 x
    const FxSplit s = fx_split(sn);
    sn = fx_mul(s, fx_split(cm), sn) << 1;
    cm = -(fx_mul(s, s) << 1);
  }
  return fx_factor(cm, sn);
}
// |z|^2 in units of 2^63
__device__ __forceinline__ fx_t fx_abs2(FxSplit x, FxSplit y) {
  const fx_t hl = fx_mad(x.h, x.l, fx_mad(y.h, y.l, 0));
  const fx_t hh = fx_mad(x.h, x.h, fx_mad(y.h, y.h, 0));
  return (hh << 1) + (hl >> 30);
}
// z + z (e^{i phi} - 1), or z + z (e^x - 1) for a real exponent
__device__ __forceinline__ FxC fx_turn(FxSplit x, FxSplit y, FxC z, int4 w) { return fx_cmul<false>(x, y, w, z); }
__device__ __forceinline__ FxC fx_grow(FxSplit x, FxSplit y, FxC z, FxSplit w) {
  return FxC{fx_mul(x, w, z.x), fx_mul(y, w, z.y)};
}

// Components of unlike scale: the products of the matrix (tables of own
// exponents e) meet at the exponent of the larger one, the other shifted down.
// (Both are calls: their code in the common path costs its small passes, which
// fetch their instructions anew in every launch, 3%.)
struct FxPair {
  FxC z0, z1;
};
static __device__ __noinline__ void fx_split_exponents(FxRow* r, int q0, int q1, int4 e) {
  const int t[4] = {q0 + 2 + e.x, q1 + 2 + e.y, q0 + 2 + e.z, q1 + 2 + e.w};
  r->qm[0] = max(t[0], t[1]);
  r->qm[1] = max(t[2], t[3]);
  for (int k = 0; k < 4; ++k) r->dm[k] = min(63, r->qm[k / 2] - t[k]);
}
static __device__ __noinline__ FxPair fx_matrix_split(FxPair z, int4 m00, int4 m01, int4 m10, int4 m11,
                                                      const int* dm) {
  auto term = [](FxC z, int4 m, int d) {  // z m 2^(-64 - d), rounded
    const FxC t = fx_cmul<false>(z, m);
    const fx_t half = (fx_t(1) << d) >> 1;
    return FxC{(t.x + half) >> d, (t.y + half) >> d};
  };
  return FxPair{cadd(term(z.z0, m00, dm[0]), term(z.z1, m01, dm[1])),
                cadd(term(z.z0, m10, dm[2]), term(z.z1, m11, dm[3]))};
}

// The interaction, matrix, interaction sequence in FP64, for a point whose
// phases are too large for the series of fx_sincos / fx_expm1.  z comes with
// exponents q and goes with exponents qm; m: the matrix, m01 and m10
// unread (zero) without coupling.  (By value: an address would keep the points
// of the common path in local memory.)
static __device__ __noinline__ FxPair fx_point_far(FxPair z, int q0, int q1, int qm0, int qm1, double lam2, double zr,
                                                   double zi, double g_uu, double g_dd, double g_ud, double2 m00,
                                                   double2 m01, double2 m10, double2 m11) {
  double2 p0 = make_double2(fx_to_double_far(z.z0.x, q0), fx_to_double_far(z.z0.y, q0));
  double2 p1 = make_double2(fx_to_double_far(z.z1.x, q1), fx_to_double_far(z.z1.y, q1));
  const double n0 = lam2 * cabs2(p0), n1 = lam2 * cabs2(p1);
  const double2 i0 = cexp_z<double>(zr, zi, g_uu * n0 + g_ud * n1);
  const double2 i1 = cexp_z<double>(zr, zi, g_dd * n1 + g_ud * n0);
  p0 = cmul(p0, i0);
  p1 = cmul(p1, i1);
  const double2 r0 = cmul(cadd(cmul(m00, p0), cmul(m01, p1)), i0);
  const double2 r1 = cmul(cadd(cmul(m11, p1), cmul(m10, p0)), i1);
  return FxPair{FxC{__double2ll_rn(ldexp(r0.x, -qm0)), __double2ll_rn(ldexp(r0.y, -qm0))},
                FxC{__double2ll_rn(ldexp(r1.x, -qm1)), __double2ll_rn(ldexp(r1.y, -qm1))}};
}

template <int N, int E, int ROWS>
__device__ __forceinline__ void row_body_fx(const RowArgs<double>& a, const BlockPos pos) {
  constexpr int T = N / E;
  constexpr int LS = N + N / E;
  constexpr int NT = 2 * T * ROWS;
  constexpr int kBits = fx_bits(stage_radix(N, E, 1));
  constexpr int kTq = fx_transform_q<N, E>();
  static_assert(NT % 32 == 0 && (T & (T - 1)) == 0, "whole warps of whole lines");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FxC* sm = reinterpret_cast<FxC*>(smem_raw);
  __shared__ uint32_t s_mx[NT / 32];
  __shared__ uint32_t s_l1[NT / 32], s_l1f[2 * ROWS], s_mxf[2 * ROWS];
  constexpr int NW = NT / 32;
  __shared__ uint32_t s_wmax[NW];
  __shared__ FxLimbs s_limb[NW];     // sums of w per warp
  __shared__ FxRow s_row[ROWS];
  __shared__ double s_w;

  const int tid = threadIdx.x;
  const int rho = tid / (2 * T);
  const int comp = (tid / T) & 1;
  const int j = tid % T;
  const int y = pos.x * ROWS + rho;
  const long long row_off = (long long)y * N;
  const bool step = a.mode == kRowStep;

  FxC v[1][E];
  int q, q_other;   // exponents of this line and of the row's other component
  bool bad, common;
  {
    const int4* __restrict__ in = reinterpret_cast<const int4*>(a.in[comp]);
    int4 w[E];
    wait_for_previous_grid();
#pragma unroll
    for (int m = 0; m < E; ++m) w[m] = in[row_off + j + m * T];
    allow_next_grid();
    if (step && a.fin == nullptr) {
      // the largest of the column pass's partial sums [comp][tile][u, w]
      uint32_t wm = 0;
      for (int i = tid; i < 2 * a.ntile; i += NT) wm = max(wm, uint32_t(__double2hiint(a.part[2 * i + 1])));
      wm = __reduce_max_sync(0xffffffffu, wm);
      if ((tid & 31) == 0) s_wmax[tid >> 5] = wm;
    }
    if (tid < 2 * ROWS) s_l1f[tid] = s_mxf[tid] = 0;
    uint32_t mx = 0, other;
#pragma unroll
    for (int m = 0; m < E; ++m) mx = fx_hi_max(mx, w[m]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (o < T) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if constexpr (T < 32) {
      other = __shfl_xor_sync(0xffffffffu, mx, T);
      __syncthreads();
    } else {
      if ((tid & 31) == 0) s_mx[tid >> 5] = mx;
      __syncthreads();
      constexpr int WL = T / 32;
      const int mine = (tid / T) * WL, theirs = ((tid / T) ^ 1) * WL;
      mx = other = 0;
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        mx = max(mx, s_mx[mine + i]);
        other = max(other, s_mx[theirs + i]);
      }
    }
    int be = fx_line_exp(mx), be_other = fx_line_exp(other);
    common = step && !a.op.diag && abs(be - be_other) <= kFxUnlike;
    if (common) be = be_other = max(be, be_other);
    // a step's densities mix the components: one bad line spoils both
    bad = be == kFxNonFinite || (step && be_other == kFxNonFinite);
    q = fx_line_q(be, 62 - kBits);
    q_other = fx_line_q(be_other, 62 - kBits);
#pragma unroll
    for (int m = 0; m < E; ++m) v[0][m] = fx_load<fx_convert(N, E)>(w[m], be, 62 - kBits);
  }
  constexpr bool kWarp = (32 % T == 0);
  constexpr int WL = T < 32 ? 0 : T / 32;  // entries of s_l1 that make up a line
  uint32_t l1 = fx_l1<E>(v[0]), l1_other = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < T) l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  if constexpr (T < 32) {
    l1_other = __shfl_xor_sync(0xffffffffu, l1, T);
  } else {
    if ((tid & 31) == 0) s_l1[tid >> 5] = l1;
    if constexpr (T == 32) __syncthreads();  // longer lines meet at the exchange
    l1 = 0;
  }
  const int line = tid / T;
  FxC* const base = sm + (comp * ROWS + rho) * LS;
  const FxLine<N, E, kWarp, true> smv(base, WL, 1, s_l1 + line * WL, l1, s_l1 + (line ^ 1) * WL, l1_other,
                                      common);
  const FxC* tw = reinterpret_cast<const FxC*>(a.twf);

  if (step) {
    int bw = 0;  // exponent of the largest partial
    if (a.fin == nullptr) {
      uint32_t wm = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) wm = max(wm, s_wmax[w]);
      bw = max(int(wm >> 20), 2);
      FxLimbs s{};
      for (int i = tid; i < 2 * a.ntile; i += NT) fx_limb_add(&s, a.part[2 * i + 1], bw);
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        const uint32_t x = __reduce_add_sync(0xffffffffu, s.l[l]);
        if ((tid & 31) == 0) s_limb[tid >> 5].l[l] = x;
      }
    }
    fft_lines<N, E, +1, 1, false, true>(v, j, smv, tw);
    if constexpr (kWarp) __syncthreads();  // the limbs of every warp
    q += kTq - smv.shift;
    q_other += kTq - smv.shift_other;
    // the row's constants, by the first thread of each row
    if (comp == 0 && j == 0) {
      double w;
      if (a.fin != nullptr) w = a.fin[2];
      else w = bw >= kFxNonFinite ? __hiloint2double(kNanHi, 0) : fx_limb_value(s_limb, NW, bw);
      // y = sqrt(1/w) 2^h by one third-order step from the FP32 root of w 2^-2h
      // in [1, 4) (FP64 operations are the longest chain of a small pass)
      const bool tiny = __double2hiint(w) < 0x100000;
      double ws = w;
      if (tiny) ws *= 0x1p108;                   // out of the subnormal range
      const int whi = __double2hiint(ws);        // still 0 when the norm is
      const int hn = ((whi >> 20) - 1023) >> 1, h = tiny ? hn - 54 : hn;
      const double wn = __hiloint2double(whi - (hn << 21), __double2loint(ws));
      const int wnh = __double2hiint(wn);
      const float y0 = rsqrtf(__int_as_float((((wnh >> 20) - 1023 + 127) << 23) | ((wnh & 0xfffff) << 3)));
      const int yb = __float_as_int(y0);
      const double ys = __hiloint2double((((yb >> 23) - 127 + 1023) << 20) | ((yb & 0x7fffff) >> 3), (yb & 7) << 29);
      const double e = __fma_rn(-(wn * ys), ys, 1.0);
      const double yw = __fma_rn(ys * e, __fma_rn(e, 0.375, 0.5), ys);
      const double lam = a.sqrt_norm * yw, y2 = yw * yw;  // lambda 2^h, 2^2h / w
      FxRow& r = s_row[rho];
      const double2 mb = a.op.mb.p[y];
      const double px = mb.x * lam, py = mb.y * lam;
      const uint32_t xh = uint32_t(__double2hiint(px)), yh = uint32_t(__double2hiint(py));
      const int be = fx_line_exp(max(xh & 0x7fffffffu, yh & 0x7fffffffu));
      // |z| <= 2^60.5, half of it (two products of a quarter) behind the
      // matrix: a factor of up to 2^62.5 leaves the headroom of any first
      // stage; a root sum square of 2^62.5 becomes 2^60, of which R points of
      // a butterfly add up to sqrt(R) 2^60
      r.pb = fx_factor(fx_from_words(xh, uint32_t(__double2loint(px)), be, 62),
                       fx_from_words(yh, uint32_t(__double2loint(py)), be, 62));
      const int qz[2] = {q, q_other};
      // the matrix tables are held as A 2^(62 - e), the products scaled by 2^-64
      r.qm[0] = q + 2 + a.me[0];
      r.qm[1] = q_other + 2 + a.me[3];
      r.split = !a.op.diag && (a.split || q != q_other);
      if (r.split) fx_split_exponents(&r, q, q_other, make_int4(a.mse[0], a.mse[1], a.mse[2], a.mse[3]));
      const double ko = a.kz[2] * y2;
      const uint32_t oh = uint32_t(__double2hiint(ko));
      const uint32_t dh[2] = {uint32_t(__double2hiint(a.kz[0] * y2)), uint32_t(__double2hiint(a.kz[1] * y2))};
      const uint32_t dl[2] = {uint32_t(__double2loint(a.kz[0] * y2)), uint32_t(__double2loint(a.kz[1] * y2))};
      uint32_t largest = oh & 0x7fffffffu;
      int raw[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        largest = max(largest, dh[k] & 0x7fffffffu);
        raw[k] = int(max(dh[k] & 0x7fffffffu, oh & 0x7fffffffu) >> 20) - 1022 + 2 * (qz[k] - h) + 129;
      }
      // |z|^2 is below 2^58 units: with shifts up to 4 no phase can leave the
      // series' range, and up to two doublings keep the shifts there for
      // phases up to 1/2
      const int twice = min(2, max(0, max(raw[0], raw[1]) - 4));
      r.twice = twice;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        // phase_i = z (g_ik lambda^2 |z_k|^2) as hi64((|z_k|^2 << sh) m) 2^-64
        const int sh = max(0, raw[k] - twice);
        const int bk = 893 - 2 * (qz[k] - h) + sh + twice;
        r.m[k][k] = fx_split((dh[k] << 1 | dl[k]) == 0 ? 0 : fx_from_words(dh[k], dl[k], bk, 62));
        r.m[1 - k][k] = fx_split(ko == 0.0 ? 0 : fx_from_words(oh, uint32_t(__double2loint(ko)), bk, 62));
        r.sh[k] = sh > 62 ? 63 : sh;  // past 62 every nonzero density goes the FP64 way
        r.q[k] = r.qm[k] + 64 + fx_line_q(be, 62) - h;
      }
      r.bad = bad || be == kFxNonFinite || int(largest >> 20) == kFxNonFinite || whi < 0x100000 ||
              (whi >> 20) == kFxNonFinite;
      if (tid == 0) s_w = w;
    }
    if (a.pops != nullptr && pos.x == 0 && tid >= NT - 32) fx_populations(a.part, a.fin, a.ntile, a.atom_num, a.pops);
    __syncthreads();
    {
      using LS0 = LineSmem<FxC, E>;
      const LS0 r0{sm + rho * LS, 0}, r1{sm + (ROWS + rho) * LS, 0};
      const int jj = tid % (2 * T);
      const FxRow& r = s_row[rho];
      const int4 pb = r.pb;
      const FxSplit m00 = r.m[0][0], m01 = r.m[0][1], m10 = r.m[1][0], m11 = r.m[1][1];
      const int sh0 = r.sh[0], sh1 = r.sh[1], twice = r.twice;
      const fx_t lim0 = fx_t(1) << max(0, 62 - sh0), lim1 = fx_t(1) << max(0, 62 - sh1);
      const bool diag = a.op.diag != 0, split = r.split, real = a.op.zi == 0.0;
      const int q0 = comp == 0 ? q : q_other, q1 = comp == 0 ? q_other : q;
      // element x = jj + m 2T at padded position pad(jj) + m kStep when 2T is
      // a multiple of E (every power of two)
      constexpr bool kFold = (2 * T) % E == 0;
      constexpr int kStep = 2 * T + (2 * T) / E;
      FxC* const b0 = r0.line(0) + LS0::pad(unsigned(jj));
      FxC* const b1 = r1.line(0) + LS0::pad(unsigned(jj));
      uint32_t h0 = E, h1 = E, g0m = 0, g1m = 0;  // L1 norms and largest values of the results
#pragma unroll 1
      for (int m = 0; m < E / 2; ++m) {
        const int x = jj + m * 2 * T;
        FxC& at0 = kFold ? b0[m * kStep] : r0.line(0)[LS0::pad(unsigned(x))];
        FxC& at1 = kFold ? b1[m * kStep] : r1.line(0)[LS0::pad(unsigned(x))];
        FxC z0 = at0, z1 = at1;
        FxSplit x0 = fx_split(z0.x), y0 = fx_split(z0.y), x1 = fx_split(z1.x), y1 = fx_split(z1.y);
        const fx_t n0 = fx_abs2(x0, y0), n1 = fx_abs2(x1, y1);
        if (n0 < lim0 && n1 < lim1) {
          const FxSplit s0 = fx_split(n0 << sh0), s1 = fx_split(n1 << sh1);
          const fx_t f0 = fx_mul(s0, m00, fx_mul(s1, m01)), f1 = fx_mul(s1, m11, fx_mul(s0, m10));
          int4 w0, w1;
          FxSplit g0, g1;
          if (real) {
            fx_t e0 = fx_expm1(f0), e1 = fx_expm1(f1);
            for (int k = 0; k < twice; ++k) {  // e^2x - 1 = 2 e + e^2
              e0 = fx_mul(fx_split(e0), fx_split(e0), e0 << 1);
              e1 = fx_mul(fx_split(e1), fx_split(e1), e1 << 1);
            }
            g0 = fx_split(e0);
            g1 = fx_split(e1);
            z0 = fx_grow(x0, y0, z0, g0);
            z1 = fx_grow(x1, y1, z1, g1);
          } else {
            w0 = fx_phase(f0, twice);
            w1 = fx_phase(f1, twice);
            z0 = fx_turn(x0, y0, z0, w0);
            z1 = fx_turn(x1, y1, z1, w1);
          }
          x0 = fx_split(z0.x), y0 = fx_split(z0.y), x1 = fx_split(z1.x), y1 = fx_split(z1.y);
          if (split) {
            const FxPair u = fx_matrix_split(FxPair{z0, z1}, __ldg(a.ms[0] + x), __ldg(a.ms[1] + x),
                                             __ldg(a.ms[2] + x), __ldg(a.ms[3] + x), r.dm);
            z0 = u.z0;
            z1 = u.z1;
          } else {
            z0 = fx_cmul<false>(x0, y0, __ldg(a.mf[0] + x), FxC{0, 0});
            z1 = fx_cmul<false>(x1, y1, __ldg(a.mf[3] + x), FxC{0, 0});
            if (!diag) {
              z0 = fx_cmul<false>(x1, y1, __ldg(a.mf[1] + x), z0);
              z1 = fx_cmul<false>(x0, y0, __ldg(a.mf[2] + x), z1);
            }
          }
          x0 = fx_split(z0.x), y0 = fx_split(z0.y), x1 = fx_split(z1.x), y1 = fx_split(z1.y);
          if (real) {
            z0 = fx_grow(x0, y0, z0, g0);
            z1 = fx_grow(x1, y1, z1, g1);
          } else {
            z0 = fx_turn(x0, y0, z0, w0);
            z1 = fx_turn(x1, y1, z1, w1);
          }
        } else {
          const double2 none = make_double2(0.0, 0.0);
          const FxPair far = fx_point_far(
              FxPair{z0, z1}, q0, q1, r.qm[0], r.qm[1], a.norm_num / s_w, a.op.zr, a.op.zi, a.g_uu, a.g_dd, a.g_ud, a.op.m[0].p[x],
              diag ? none : a.op.m[1].p[x], diag ? none : a.op.m[2].p[x], a.op.m[3].p[x]);
          z0 = far.z0;
          z1 = far.z1;
        }
        z0 = fx_cmul<false>(z0, pb);
        z1 = fx_cmul<false>(z1, pb);
        const uint32_t a0 = uint32_t(abs(int(z0.x >> 32))), b0h = uint32_t(abs(int(z0.y >> 32)));
        const uint32_t a1 = uint32_t(abs(int(z1.x >> 32))), b1h = uint32_t(abs(int(z1.y >> 32)));
        h0 += a0 + b0h;
        h1 += a1 + b1h;
        g0m = max(g0m, max(a0, b0h));
        g1m = max(g1m, max(a1, b1h));
        at0 = z0;
        at1 = z1;
      }
      h0 = (h0 >> 12) + 1;
      h1 = (h1 >> 12) + 1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (o < 2 * T) {
          h0 += __shfl_xor_sync(0xffffffffu, h0, o);
          h1 += __shfl_xor_sync(0xffffffffu, h1, o);
          g0m = max(g0m, __shfl_xor_sync(0xffffffffu, g0m, o));
          g1m = max(g1m, __shfl_xor_sync(0xffffffffu, g1m, o));
        }
      if (tid % (2 * T < 32 ? 2 * T : 32) == 0) {
        atomicAdd(&s_l1f[2 * rho], h0);
        atomicAdd(&s_l1f[2 * rho + 1], h1);
        atomicMax(&s_mxf[2 * rho], g0m);
        atomicMax(&s_mxf[2 * rho + 1], g1m);
      }
    }
    __syncthreads();
    bad = s_row[rho].bad;
    q = s_row[rho].q[comp];
    FxLine<N, E, kWarp, false> fwd(base, 1, 1, &s_l1f[2 * rho + comp]);
    fwd.pre = fx_pre(s_mxf[2 * rho + comp], kBits);
    fft_lines<N, E, -1, 1, true, false>(v, j, fwd, tw);
    q += kTq - fwd.shift;
  } else {
    if (a.mode == kRowForward) fft_lines<N, E, -1, 1>(v, j, smv, tw);
    else fft_lines<N, E, +1, 1>(v, j, smv, tw);
    q += kTq - smv.shift;
    if (a.scale != 1.0) {
      const FxScale s = fx_scale(a.scale);
#pragma unroll
      for (int m = 0; m < E; ++m) {
        v[0][m].x = fx_mul(fx_split(v[0][m].x), s.m);
        v[0][m].y = fx_mul(fx_split(v[0][m].y), s.m);
      }
      q += 64 + s.e;
      bad = bad || !s.finite;
    }
  }
  int4* out = reinterpret_cast<int4*>(a.out[comp]);
  auto write = [&](auto form) {
#pragma unroll
    for (int m = 0; m < E; ++m) out[row_off + j + m * T] = fx_words<decltype(form)::value, fx_convert(N, E)>(v[0][m], q);
  };
  const FxOut form = fx_out(bad, q);
  if (form == kFxNear) write(std::integral_constant<FxOut, kFxNear>{});
  else if (form == kFxBad) write(std::integral_constant<FxOut, kFxBad>{});
  else write(std::integral_constant<FxOut, kFxFar>{});
}

template <int N, int E, int ROWS, int MINB>
__global__ void __launch_bounds__(2 * (N / E) * ROWS, MINB)
row_kernel_fx(const RowArgs<double> a) {
  row_body_fx<N, E, ROWS>(a, grid_pos());
}
template <int N, int E, int ROWS, int MINB>
__global__ void __launch_bounds__(2 * (N / E) * ROWS, MINB)
row_kernel_fx_grouped(const RowArgs<double>* __restrict__ args) {
  row_body_fx<N, E, ROWS>(args[blockIdx.y], grid_pos());
}

}  // namespace sgpe
