// Line transforms of the projection with the levels paired and the FFT passes
// run between registers and one in-place shared-memory line.
//
// The earlier pencils (pencil.cuh, xreg.cuh, xreg4.cuh) stage a tile in shared
// memory, transform it and stage it out again: 5 to 6 trips through shared
// memory per value and, where the tile fills the SM, one CTA whose load,
// transform and store phases follow one another.  Here
//  * the first pass loads its butterfly's rows straight from global memory
//    into registers and the last one stores its outputs straight to global
//    memory, so a line crosses shared memory once per pass boundary (twice for
//    three passes) and needs no staging tile;
//  * two adjacent levels of a real field are the real and imaginary part of one
//    complex line of length nx, so the forward transform needs no half-length
//    split with its twiddles and the inverse one no pre-process: one Hermitian
//    add and subtract in the pass that touches global memory;
//  * a forward transform decimates in time (digit-reversed rows in, natural
//    wavenumbers out) and an inverse one in frequency (the transpose), so every
//    pass works in place: one buffer per line, no ping-pong, and several CTAs
//    per SM, whose phases overlap.
// What bounds them: the latency of loads, then the first-level cache's line
// accesses (at 1024 points, 15 warps per SM in single precision and 8 in double:
// 4 to 5 long-scoreboard stalls an issue, that cache 47 to 54% busy, DRAM 19 to
// 38%); at small grids the latency of the three passes.  Measured per launch against the best
// earlier form (device time, us):
//   512 x 512 x 64 double:    x 474 -> 246 and back 551 -> 350, y 186 -> 117
//                             and back 203 -> 127
//   1024 x 1024 x 80 single:  x back 1600 -> 1040, y 428 -> 372 and back 376 -> 340
//   512 x 512 x 64 single:    x 158 -> 135 and back 261 -> 172
//
// Lanes: consecutive threads take consecutive columns (level pairs, or levels
// in the y kernels), then consecutive butterflies of a line.  Positions in the
// buffer are padded by one slot every r[0] positions when r[0] is a power of
// two, which spreads the adjacent-position pass over the banks.
#pragma once
#include <type_traits>

#include "fft.cuh"
#include "zfft.h"

namespace ob {

__host__ __device__ constexpr int zlog2(int c) { return c == 1 ? 0 : 1 + zlog2(c / 2); }

// The thread index, opaque to the optimiser: each pass computes its own
// indices instead of keeping every radix's across all passes in registers.
__device__ __forceinline__ int ztid() {
  int t = threadIdx.x;
  asm volatile("" : "+r"(t));
  return t;
}

__device__ __forceinline__ int zphys(const ZPlan& p, int pos) { return pos + (pos >> p.sh); }

// first input row of first-pass butterfly b (digits j1, j2, .. of b reversed)
__device__ __forceinline__ int zrev(const ZPlan& p, int b) {
  if (p.np == 2) return b;
  int q = p.dr[1].div(b);
  int acc = b - q * p.r[1];
  if (p.np == 3) return acc * p.r[2] + q;
  const int q2 = p.dr[2].div(q);
  acc = acc * p.r[2] + (q - q2 * p.r[2]);
  return acc * p.r[3] + q2;
}

// ---- further small DFTs --------------------------------------------------------
// N1 N2 points with N1 and N2 coprime, by Good's prime-factor index map: no
// twiddles between the two stages.
template <class T, int N1, int N2, bool INV>
__device__ __forceinline__ void dft_pfa(cplx<T>* v) {
  constexpr int N = N1 * N2;
  cplx<T> w[N];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) {
    cplx<T> a[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) a[n1] = v[(N2 * n1 + N1 * n2) % N];
    dft_small<T, N1, INV>(a);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) w[k1 * N2 + n2] = a[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) {
    dft_small<T, N2, INV>(w + k1 * N2);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      // the k with k = k1 (mod N1) and k = k2 (mod N2)
      int k = 0;
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c % N1 == k1 && c % N2 == k2) k = c;
      v[k] = w[k1 * N2 + k2];
    }
  }
}

template <class T, bool INV>
__device__ __forceinline__ void dft9(cplx<T>* v) {
  const T c1 = (T)0.76604444311897803520, s1 = (T)0.64278760968653932632;  // 2 pi / 9
  const T c2 = (T)0.17364817766693034885, s2 = (T)0.98480775301220805937;  // 4 pi / 9
  const T c4 = (T)-0.93969262078590838405, s4 = (T)0.34202014332566873304; // 8 pi / 9
  cplx<T> a[3], b[3], c[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a[i] = v[3 * i];
    b[i] = v[3 * i + 1];
    c[i] = v[3 * i + 2];
  }
  dft3<T, INV>(a);
  dft3<T, INV>(b);
  dft3<T, INV>(c);
  b[1] = twc<T, INV>(b[1], c1, s1);
  b[2] = twc<T, INV>(b[2], c2, s2);
  c[1] = twc<T, INV>(c[1], c2, s2);
  c[2] = twc<T, INV>(c[2], c4, s4);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cplx<T> t[3] = {a[k], b[k], c[k]};
    dft3<T, INV>(t);
    v[k] = t[0];
    v[k + 3] = t[1];
    v[k + 6] = t[2];
  }
}

template <class T, int R, bool INV>
__device__ __forceinline__ void zdft(cplx<T>* v) {
  if constexpr (R == 6) dft_pfa<T, 2, 3, INV>(v);
  else if constexpr (R == 9) dft9<T, INV>(v);
  else if constexpr (R == 10) dft_pfa<T, 2, 5, INV>(v);
  else if constexpr (R == 12) dft_pfa<T, 3, 4, INV>(v);
  else if constexpr (R == 15) dft_pfa<T, 3, 5, INV>(v);
  else dft_small<T, R, INV>(v);
}

// Radices: of the passes that touch global memory (z_edge: a line's
// adjacent pass; z_pair: even, the pass that pairs wavenumbers k and N - k) and
// of the passes in between.
template <class F>
__device__ __forceinline__ void z_edge(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
  }
}
template <class F>
__device__ __forceinline__ void z_mid(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 12: f(std::integral_constant<int, 12>{}); break;
    case 15: f(std::integral_constant<int, 15>{}); break;
    case 16: f(std::integral_constant<int, 16>{}); break;
  }
}
template <class F>
__device__ __forceinline__ void z_pair(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
  }
}

// tw: for pass i the twiddles of its elements j = 1 .. r[i]-1 at [S[i] - 1 +
// (j - 1) S[i] + k], so the butterflies of a warp read neighbouring entries (a
// single table read at j k apart costs the first-level cache a line per lane).
template <class T, bool INV>
__device__ __forceinline__ cplx<T> ztw(cplx<T> a, const cplx<T>* __restrict__ tw, int i) {
  cplx<T> w;
  if constexpr (sizeof(T) == 4) {
    const float2 f = __ldg(reinterpret_cast<const float2*>(tw) + i);
    w.x = f.x;
    w.y = f.y;
  } else {
    const double2 f = __ldg(reinterpret_cast<const double2*>(tw) + i);
    w.x = f.x;
    w.y = f.y;
  }
  if (INV) w.y = -w.y;
  return mul(a, w);
}

// A pass between the first and the last, in place (forward: twiddles before
// the DFT; inverse: after it).  buf: RY lines of NP slots of C columns, slots st
// and lines rs elements apart (by default packed).
template <class T, int C, bool INV>
__device__ __forceinline__ void z_mid_pass(const ZPlan& p, int i, cplx<T>* buf, int RY,
                                           const cplx<T>* __restrict__ tw, int st = C,
                                           int rs = 0) {
  if (!rs) rs = p.NP * C;
  constexpr int LC = zlog2(C);
  z_mid(p.r[i], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int S = p.S[i], nb = p.nb[i];
    const int Sp = (S + (S >> p.sh)) * st;
    const int tot = RY * nb * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      const int c = e & (C - 1);
      int b = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dnb[i].div(b);
        b -= row * nb;
      }
      const int m = p.dS[i].div(b);
      const int k = b - m * S;
      cplx<T>* q = buf + row * rs + zphys(p, m * (S * R) + k) * st + c;
      cplx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = q[j * Sp];
      const cplx<T>* tk = tw + (S - 1 + k);
      if (!INV) {
#pragma unroll
        for (int j = 1; j < R; ++j) v[j] = ztw<T, false>(v[j], tk, (j - 1) * S);
      }
      zdft<T, R, INV>(v);
      if (INV) {
#pragma unroll
        for (int j = 1; j < R; ++j) v[j] = ztw<T, true>(v[j], tk, (j - 1) * S);
      }
#pragma unroll
      for (int j = 0; j < R; ++j) q[j * Sp] = v[j];
    }
  });
}

// The adjacent-position pass of a forward transform: load(row, c, n, v) gives
// the butterfly's inputs of rows n, n + N / R, ..
template <class T, int C, class Load>
__device__ __forceinline__ void z_first_fwd(const ZPlan& p, cplx<T>* buf, int RY, Load&& load,
                                            int st = C, int rs = 0) {
  if (!rs) rs = p.NP * C;
  constexpr int LC = zlog2(C);
  z_edge(p.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nb = p.nb[0];
    const int tot = RY * nb * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      const int c = e & (C - 1);
      int b = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dnb[0].div(b);
        b -= row * nb;
      }
      cplx<T> v[R];
      load(rc, row, c, zrev(p, b), nb, v);
      zdft<T, R, false>(v);
      cplx<T>* q = buf + row * rs + zphys(p, b * R) * st + c;
#pragma unroll
      for (int j = 0; j < R; ++j) q[j * st] = v[j];
    }
  });
}

// The adjacent-position pass of an inverse transform: store(row, n, step, q)
// reads the butterfly's inputs q[j C], transforms them and takes output rows
// n, n + step, ..
template <class T, int C, class Store>
__device__ __forceinline__ void z_last_inv(const ZPlan& p, const cplx<T>* buf, int RY,
                                           Store&& store, int st = C, int rs = 0) {
  if (!rs) rs = p.NP * C;
  constexpr int LC = zlog2(C);
  z_edge(p.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nb = p.nb[0];
    const int tot = RY * nb * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      const int c = e & (C - 1);
      int b = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dnb[0].div(b);
        b -= row * nb;
      }
      store(rc, row, zrev(p, b), nb, buf + row * rs + zphys(p, b * R) * st + c);
    }
  });
}

// ---- level pairs -----------------------------------------------------------------
// Two adjacent levels of one field, the first at p; vec: one access for both, which
// wants p on a multiple of its size (zpairs); two: the second level exists.
template <class TS>
struct __align__(2 * sizeof(TS)) pair2 {
  TS a, b;
};
template <class TS>
__device__ __forceinline__ pair2<TS> ldpair(const TS* p, bool vec, bool two) {
  pair2<TS> r;
  if (vec) {
    r = *reinterpret_cast<const pair2<TS>*>(p);
  } else {
    r.a = p[0];
    r.b = two ? p[1] : (TS)0;
  }
  return r;
}
template <class TS>
__device__ __forceinline__ void stpair(TS* p, TS a, TS b, bool vec, bool two) {
  if (vec) {
    pair2<TS> r;
    r.a = a;
    r.b = b;
    *reinterpret_cast<pair2<TS>*>(p) = r;
  } else {
    p[0] = a;
    if (two) p[1] = b;
  }
}
template <class T>
struct cpair {
  cplx<T> a, b;
};
template <class T>
__device__ __forceinline__ cpair<T> ldcpair(const cplx<T>* p, bool vec, bool two,
                                            bool one = true) {
  cpair<T> r;
  if constexpr (sizeof(T) == 4) {
    if (vec) {
      const float4 f = *reinterpret_cast<const float4*>(p);
      r.a.x = f.x;
      r.a.y = f.y;
      r.b.x = f.z;
      r.b.y = f.w;
      return r;
    }
  }
  r.a = one ? p[0] : mk<T>((T)0, (T)0);
  r.b = two ? p[1] : mk<T>((T)0, (T)0);
  return r;
}
template <class T>
__device__ __forceinline__ void stcpair(cplx<T>* p, cplx<T> a, cplx<T> b, bool vec, bool two) {
  if constexpr (sizeof(T) == 4) {
    if (vec) {
      *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
      return;
    }
  }
  p[0] = a;
  if (two) p[1] = b;
}

// A column weight in the transform's type with what its rounding to float
// leaves: products with it round once, as products formed in double do.
template <class T>
struct zwt {
  T h, l;
};
template <class T>
__device__ __forceinline__ zwt<T> mkwt(double w) {
  zwt<T> r;
  r.h = (T)w;
  r.l = sizeof(T) == 4 ? (T)(w - (double)r.h) : (T)0;
  return r;
}
template <class T>
__device__ __forceinline__ T wmul(zwt<T> w, T a) {
  if constexpr (sizeof(T) == 4) return fmaf(a, w.h, a * w.l);
  else return a * w.h;
}
// ru wu - rl wl; in single precision the rounding error of the product that
// is subtracted is recovered by an FMA, so the difference is as good as one
// formed in double and rounded
template <class T>
__device__ __forceinline__ T wdiff(zwt<T> ru, T wu, zwt<T> rl, T wl) {
  if constexpr (sizeof(T) == 4) {
    const float q = wl * rl.h;
    const float e = fmaf(-wl, rl.h, q);
    const float r = fmaf(wu, ru.h, -q);
    return r + (e + fmaf(wu, ru.l, -(wl * rl.l)));
  } else {
    return srn(mrn(ru.h, wu), mrn(rl.h, wl));
  }
}
// the same of values with what their own rounding left, which counts where they
// nearly cancel
template <class T>
struct zval {
  T h, l;
};
template <class T>
__device__ __forceinline__ T wdiff(zwt<T> ru, zval<T> wu, zwt<T> rl, zval<T> wl) {
  if constexpr (sizeof(T) == 4) {
    const float q = wl.h * rl.h;
    const float e = fmaf(-wl.h, rl.h, q);
    const float r = fmaf(wu.h, ru.h, -q);
    const float t = fmaf(wu.l, ru.h, -(wl.l * rl.h));
    return r + (e + fmaf(wu.h, ru.l, fmaf(-wl.h, rl.l, t)));
  } else {
    return wdiff(ru, wu.h, rl, wl.h);
  }
}

// Provisional stage w: w + sdt b (integrator.py:483-490).  Single precision: the
// sum in two floats, so that the flux difference of its values is as good as in
// double.  Rounded to one float first, it would add an ulp of w over dz to the
// source, more than all its other roundings where w is large against sdt b.
__device__ __forceinline__ zval<double> zstage(double w, zwt<double> sdt, double b) {
  return {arn(w, mrn(sdt.h, b)), 0.0};
}
__device__ __forceinline__ zval<float> zstage(float w, zwt<float> sdt, float b) {
  const float p = mrn(sdt.h, b);
  const float e = fmaf(sdt.l, b, fmaf(sdt.h, b, -p));  // sdt b - p
  const float s = arn(w, p);
  const float x = srn(s, w);                           // the part of p that s took
  return {s, arn(arn(srn(w, srn(s, x)), srn(p, x)), e)};
}
// the same rounded once (an infinite sum has no remainder)
template <class T>
__device__ __forceinline__ T zstage1(T w, zwt<T> sdt, T b) {
  const zval<T> s = zstage(w, sdt, b);
  if (sizeof(T) == 8 || isnan(s.l)) return s.h;
  return s.h + s.l;
}

// Level pairs per CTA.  A warp's access costs the first-level cache one pass
// per 128-byte line it touches, and these kernels are bound by those passes
// before they are by memory, so a row's run is as long as shared memory allows:
// 16 levels in single precision and 8 in double, 64 bytes of a state field and
// a whole line of a spectrum.
template <class T>
__host__ __device__ constexpr int zx_pairs() { return sizeof(T) == 4 ? 8 : 4; }
// Columns (levels) per CTA of the y kernels: 64-byte runs of a spectrum, or half
// of that for two long lines per column.
template <class T>
__host__ __device__ constexpr int zy_cols() { return sizeof(T) == 4 ? 8 : 4; }

constexpr int kZThreads = 256;
// threads of an x block and blocks per SM its registers must allow: 24 warps of
// 80 registers in single precision, 16 of 128 in double, some of whose wider
// butterflies spill; without spills (128 and 168 registers) the fewer warps cost
// more (512 x 512 x 64, back along x: 194 against 172 us, 362 against 350)
template <class T>
__host__ __device__ constexpr int zx_threads() { return sizeof(T) == 4 ? 256 : 128; }
template <class T>
__host__ __device__ constexpr int zx_blocks() { return sizeof(T) == 4 ? 3 : 4; }

// Splits the wavenumbers of a paired last pass into the two levels' half
// spectra and stores them (sum: adds them): v1 = F[t1 + Q j], v2 = F[t2 + Q j],
// t2 = Q - t1 (or t1 = 0, t2 = Q / 2, which pair with themselves).
template <class T, int R>
__device__ __forceinline__ void z_split_store(const ZPlan& p, int s, bool has2, cplx<T>* v1,
                                              cplx<T>* v2, cplx<T>* out, int kst, bool vec,
                                              bool two, bool sum) {
  const int t1 = s, t2 = s ? p.Q - s : p.Q / 2;
  const T h = (T)0.5;
  // what the outputs hold already, in one batch
  cpair<T> o1[R / 2], o2[R / 2];
  if (sum) {
#pragma unroll
    for (int j = 0; j < R / 2; ++j) o1[j] = ldcpair(out + (t1 + p.Q * j) * kst, vec, two);
    if (has2) {
#pragma unroll
      for (int j = 0; j < R / 2; ++j) o2[j] = ldcpair(out + (t2 + p.Q * j) * kst, vec, two);
    }
  }
  auto put = [&](int k, cplx<T> f, cplx<T> g, const cpair<T>& o) {
    cplx<T> a = mk<T>(h * (f.x + g.x), h * (f.y - g.y));
    cplx<T> b = mk<T>(h * (f.y + g.y), h * (g.x - f.x));
    if (sum) {
      a = add(a, o.a);
      b = add(b, o.b);
    }
    stcpair(out + k * kst, a, b, vec, two);
  };
  if (s) {
#pragma unroll
    for (int j = 0; j < R / 2; ++j) put(t1 + p.Q * j, v1[j], v2[R - 1 - j], o1[j]);
#pragma unroll
    for (int j = 0; j < R / 2; ++j) put(t2 + p.Q * j, v2[j], v1[R - 1 - j], o2[j]);
  } else {
#pragma unroll
    for (int j = 0; j < R / 2; ++j) put(p.Q * j, v1[j], v1[(R - j) % R], o1[j]);
    cpair<T> on{};
    if (sum) on = ldcpair(out + (p.N / 2) * kst, vec, two);
    put(p.N / 2, v1[R / 2], v1[R / 2], on);
    if (has2) {
#pragma unroll
      for (int j = 0; j < R / 2; ++j) put(t2 + p.Q * j, v2[j], v2[R - 1 - j], o2[j]);
    }
  }
}

// transforms one butterfly of the first inverse pass's values x and
// stores it with its twiddles.
template <class T, int R, int C>
__device__ __forceinline__ void z_first_bfly_inv(const ZPlan& p, cplx<T>* line, int t,
                                                 const cplx<T>* __restrict__ tw, cplx<T>* x,
                                                 int st = C) {
  zdft<T, R, true>(x);
  const int Qp = (p.Q + (p.Q >> p.sh)) * st;
  cplx<T>* o = line + zphys(p, t) * st;
  o[0] = x[0];
#pragma unroll
  for (int j = 1; j < R; ++j)
    o[j * Qp] = ztw<T, true>(x[j], tw + (p.Q - 1 + t), (j - 1) * p.Q);
}

// reads and transforms one butterfly of the last forward pass
template <class T, int R, int C>
__device__ __forceinline__ void z_last_bfly(const ZPlan& p, const cplx<T>* line, int t,
                                            const cplx<T>* __restrict__ tw, cplx<T>* v,
                                            int st = C) {
  const int Qp = (p.Q + (p.Q >> p.sh)) * st;
  const cplx<T>* q = line + zphys(p, t) * st;
#pragma unroll
  for (int j = 0; j < R; ++j) v[j] = q[j * Qp];
#pragma unroll
  for (int j = 1; j < R; ++j) v[j] = ztw<T, false>(v[j], tw + (p.Q - 1 + t), (j - 1) * p.Q);
  zdft<T, R, false>(v);
}

// Forward x transforms; RL: the line's last radix (a switch over it here costs
// the compiler the registers); pairs: level pairs in one access each (zpairs).
// grid = (ceil(nz / levels), ceil(ny / RY)); dynamic shared memory: RY lines.
template <class T, class TS, int MODE, int RL>
__global__ void __launch_bounds__(zx_threads<T>(), zx_blocks<T>()) k_zfx(
    const __grid_constant__ ZPlan p, GridK g, int RY, bool pairs, const TS* __restrict__ u,
    const TS* __restrict__ v, const TS* __restrict__ w, const TS* __restrict__ bh, double sdt,
    const double* __restrict__ rho, const double* __restrict__ rhoh, const T* __restrict__ kx,
    const cplx<T>* __restrict__ tw, cplx<T>* __restrict__ X0, cplx<T>* __restrict__ X1) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int C = zx_pairs<T>();
  constexpr int LC = zlog2(C);
  cplx<T>* b0 = reinterpret_cast<cplx<T>*>(smem_dyn);
  const int ny = g.ny, nz = g.nz;
  const int y0 = blockIdx.y * RY;
  // line sets, a block each: rho u with D w, and rho v
  const int sets = MODE == ZFX_FIELDS && !v ? 1 : 2;
  const int chunk = blockIdx.x / sets, set = blockIdx.x - chunk * sets;
  const int z = (chunk * C + (threadIdx.x & (C - 1))) * 2;  // the thread's first level
  const bool on = z < nz, two = z + 1 < nz, vec = pairs;
  const int rows = min(RY, ny - y0);
  const int xs = ny * nz, ws = ny * (nz + 1);
  zwt<T> ra{}, rb{}, f0{}, f1{}, f2{};
  if (on && MODE != ZFX_FIELDS) {
    const double id = 1.0 / g.dz;
    ra = mkwt<T>(rho[z]);
    rb = mkwt<T>(two ? rho[z + 1] : 0.0);
    f0 = mkwt<T>(rhoh[z] * id);
    f1 = mkwt<T>(rhoh[z + 1] * id);
    f2 = mkwt<T>(two ? rhoh[z + 2] * id : 0.0);
  }
  const zwt<T> sd = mkwt<T>(sdt);
  // rows of a field at this thread's level pair, weighted
  auto field = [&](const TS* f, bool weigh) {
    return [=](auto rc, int row, int c, int n, int step, cplx<T>* r) {
      constexpr int R = decltype(rc)::value;
      if (!on || row >= rows) return;
      const TS* q = f + (n * ny + y0 + row) * nz + z;
      pair2<TS> a[R];
#pragma unroll
      for (int j = 0; j < R; ++j) a[j] = ldpair(q + j * step * xs, vec, two);
#pragma unroll
      for (int j = 0; j < R; ++j)
        r[j] = weigh ? mk<T>(wmul(ra, (T)a[j].a), wmul(rb, (T)a[j].b))
                     : mk<T>((T)a[j].a, (T)a[j].b);
    };
  };
  // vertical flux divergence of w (STAGE: of w + sdt b_half)
  auto flux = [&]() {
    return [=](auto rc, int row, int c, int n, int step, cplx<T>* r) {
      constexpr int R = decltype(rc)::value;
      if (!on || row >= rows) return;
      const int o = (n * ny + y0 + row) * (nz + 1) + z;
      T w0[R], w1[R], w2[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const TS* q = w + o + j * step * ws;
        w0[j] = (T)q[0];
        w1[j] = (T)q[1];
        w2[j] = two ? (T)q[2] : (T)0;
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (MODE == ZFX_STAGE) {
          const TS* q = bh + o + j * step * ws;
          const zval<T> s0 = zstage(w0[j], sd, (T)q[0]), s1 = zstage(w1[j], sd, (T)q[1]);
          const zval<T> s2 = zstage(w2[j], sd, two ? (T)q[2] : (T)0);
          r[j] = mk<T>(wdiff(f1, s1, f0, s0), two ? wdiff(f2, s2, f1, s1) : (T)0);
        } else {
          r[j] = mk<T>(wdiff(f1, w1[j], f0, w0[j]), two ? wdiff(f2, w2[j], f1, w1[j]) : (T)0);
        }
      }
    };
  };
  // A set's lines in turn: rho u (X0 = i kx' times it), then D w, added to X0: the
  // thread reads back what it stored (from L2), which costs less than a second
  // line of shared memory, hence half the blocks.
#pragma unroll
  for (int run = 0; run < (MODE == ZFX_FIELDS ? 1 : 2); ++run) {
    const bool sum = run == 1;
    if (sum && set) return;
    const bool grad = MODE != ZFX_FIELDS && set == 0 && !sum;  // times i kx'
    cplx<T>* out = set == 0 ? X0 : X1;
    if (run) __syncthreads();
    if (MODE != ZFX_FIELDS && sum) z_first_fwd<T, C>(p, b0, RY, flux());
    else z_first_fwd<T, C>(p, b0, RY, field(set ? v : u, MODE != ZFX_FIELDS));
    __syncthreads();
#pragma unroll 1
    for (int i = 1; i + 1 < p.np; ++i) {
      z_mid_pass<T, C, false>(p, i, b0, RY, tw);
      __syncthreads();
    }
    constexpr int R = RL;
    const int tot = RY * p.ns * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      int s = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dns.div(s);
        s -= row * p.ns;
      }
      if (!on || row >= rows) continue;
      const size_t lo = (size_t)row * p.NP * C + (e & (C - 1));
      const bool has2 = s || !(p.Q & 1);
      cplx<T> v1[R], v2[R];
      z_last_bfly<T, R, C>(p, b0 + lo, s, tw, v1);
      if (has2) z_last_bfly<T, R, C>(p, b0 + lo, s ? p.Q - s : p.Q / 2, tw, v2);
      if (grad) {  // before the split: the signed kx' keeps the line Hermitian
        const int t2 = s ? p.Q - s : p.Q / 2;
#pragma unroll
        for (int j = 0; j < R; ++j) v1[j] = ik(__ldg(kx + s + p.Q * j), v1[j]);
        if (has2) {
#pragma unroll
          for (int j = 0; j < R; ++j) v2[j] = ik(__ldg(kx + t2 + p.Q * j), v2[j]);
        }
      }
      z_split_store<T, R>(p, s, has2, v1, v2, out + (y0 + row) * nz + z, xs, vec, two, sum);
    }
  }
}

// Inverse x transforms with the velocity correction, a line per block: i kx' phi~
// (u), psi~ (v) and
//  * where the potential is not stored, the level difference of phi~ (w), taken in
//    the spectrum: no halo level, no difference of rounded potentials;
//  * where it is, phi~ itself, w corrected by the differences of the values
//    stored (so a defect correction, which sees the state, also corrects their
//    rounding).  Its blocks overlap by the level below their first interface:
//    2 C levels, 2 C - 1 interfaces.
template <class T, class TS, int MODE, int RL>
__global__ void __launch_bounds__(zx_threads<T>(), zx_blocks<T>()) k_zix(
    const __grid_constant__ ZPlan p, GridK g, int RY, bool pairs, const cplx<T>* __restrict__ S1,
    const cplx<T>* __restrict__ S2, const T* __restrict__ kx, const cplx<T>* __restrict__ tw,
    const TS* u_in, const TS* v_in, const TS* w_in, const TS* __restrict__ bh, double sdt,
    TS* u_out, TS* v_out, TS* w_out, TS* phi_out) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int C = zx_pairs<T>();
  constexpr int LC = zlog2(C);
  cplx<T>* b0 = reinterpret_cast<cplx<T>*>(smem_dyn);
  const int ny = g.ny, nz = g.nz;
  const int y0 = blockIdx.y * RY;
  // lines 0: d/dx (from S1), 1: d/dy (from S2), 2: d/dz or phi (from S1): the
  // lines of a tile run side by side, so the tile's spectra still come from L2
  const int runs = MODE == ZIX_FIELDS ? (S2 ? 2 : 1) : 3;
  const int chunks = (nz + 2 * C - 1) / (2 * C);
  int chunk = blockIdx.x / runs, run = blockIdx.x - chunk * runs;
  if (MODE != ZIX_FIELDS && chunk >= chunks) {  // the potential's further blocks
    chunk = blockIdx.x - 2 * chunks;
    run = 2;
  }
  const bool pot = MODE != ZIX_FIELDS && MODE != ZIX_GRAD && run == 2 && phi_out;
  const int c = threadIdx.x & (C - 1);
  const int z = pot ? chunk * (2 * C - 1) - 1 + 2 * c : (chunk * C + c) * 2;
  const bool on = z < nz, two = z + 1 < nz, one = z >= 0;
  const bool vec = pairs && !pot;
  const int rows = min(RY, ny - y0);
  const int xs = ny * nz, ws = ny * (nz + 1);
  const T idz = (T)(1.0 / g.dz);
  const zwt<T> sd = mkwt<T>(sdt);

    const cplx<T>* src = run == 1 ? S2 : S1;
    const bool gx = MODE != ZIX_FIELDS && run == 0;
    const bool gz = MODE != ZIX_FIELDS && run == 2 && !pot;
    // First pass: wavenumbers t + Q j and their mirrors N - k of butterflies
    // t1 and t2, from the half spectra of the two levels.
    {
      constexpr int R = RL;
      const int tot = RY * p.ns * C;
      for (int e = ztid(); e < tot; e += blockDim.x) {
        int s = e >> LC, row = 0;
        if (RY > 1) {
          row = p.dns.div(s);
          s -= row * p.ns;
        }
        if (!on || row >= rows) continue;
        const bool has2 = s || !(p.Q & 1);
        const int t1 = s, t2 = s ? p.Q - s : p.Q / 2;
        const cplx<T>* q = src + (y0 + row) * nz + z;
        // loads in one batch: R / 2 wavenumbers of each butterfly
        cpair<T> x1[R / 2], x2[R / 2], xn;
#pragma unroll
        for (int j = 0; j < R / 2; ++j) x1[j] = ldcpair(q + (t1 + p.Q * j) * xs, vec, two, one);
        if (has2) {
#pragma unroll
          for (int j = 0; j < R / 2; ++j) x2[j] = ldcpair(q + (t2 + p.Q * j) * xs, vec, two, one);
        }
        if (!s) xn = ldcpair(q + (p.N / 2) * xs, vec, two, one);
        if (gz) {
          // the difference to the level below (none at the surface)
          auto below = [&](int k, cpair<T>& x) {
            cplx<T> h = x.a;
            if (z > 0) h = q[k * xs - 1];
            x.b = scl(sub(x.b, x.a), idz);
            x.a = scl(sub(x.a, h), idz);
          };
#pragma unroll
          for (int j = 0; j < R / 2; ++j) below(t1 + p.Q * j, x1[j]);
          if (has2) {
#pragma unroll
            for (int j = 0; j < R / 2; ++j) below(t2 + p.Q * j, x2[j]);
          }
          if (!s) below(p.N / 2, xn);
        }
        cplx<T> v1[R], v2[R];
        auto get = [&](int k, const cpair<T>& x, cplx<T>& f, cplx<T>& m) {
          f = mk<T>(x.a.x - x.b.y, x.a.y + x.b.x);
          m = mk<T>(x.a.x + x.b.y, x.b.x - x.a.y);
          if (gx) {
            const T kk = __ldg(kx + k);
            f = ik(kk, f);
            m = ik(-kk, m);
          }
        };
        if (s) {
#pragma unroll
          for (int j = 0; j < R / 2; ++j) {
            get(t1 + p.Q * j, x1[j], v1[j], v2[R - 1 - j]);
            get(t2 + p.Q * j, x2[j], v2[j], v1[R - 1 - j]);
          }
        } else {
          // wavenumber 0 and the Nyquist one have no imaginary part (and no
          // x derivative)
          v1[0] = gx ? mk<T>((T)0, (T)0) : mk<T>(x1[0].a.x, x1[0].b.x);
          v1[R / 2] = gx ? mk<T>((T)0, (T)0) : mk<T>(xn.a.x, xn.b.x);
#pragma unroll
          for (int j = 1; j < R / 2; ++j) get(p.Q * j, x1[j], v1[j], v1[R - j]);
          if (has2) {
#pragma unroll
            for (int j = 0; j < R / 2; ++j) get(t2 + p.Q * j, x2[j], v2[j], v2[R - 1 - j]);
          }
        }
        cplx<T>* line = b0 + (size_t)row * p.NP * C + (e & (C - 1));
        z_first_bfly_inv<T, R, C>(p, line, t1, tw, v1);
        if (has2) z_first_bfly_inv<T, R, C>(p, line, t2, tw, v2);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = p.np - 2; i >= 1; --i) {
      z_mid_pass<T, C, true>(p, i, b0, RY, tw);
      __syncthreads();
    }
    // Last pass.  The full-level lines: out = in - line, or the line itself.
    if (run < 2) {
      const TS* in = run == 0 ? u_in : v_in;
      TS* out = run == 0 ? u_out : v_out;
      z_last_inv<T, C>(p, b0, RY, [&](auto rc, int row, int n, int step, const cplx<T>* q) {
        constexpr int R = decltype(rc)::value;
        if (!on || row >= rows) return;
        const int o = (n * ny + y0 + row) * nz + z;
        pair2<TS> a[R];
        if (MODE != ZIX_FIELDS && MODE != ZIX_GRAD) {
#pragma unroll
          for (int j = 0; j < R; ++j) a[j] = ldpair(in + o + j * step * xs, vec, two);
        }
        cplx<T> x[R];
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = q[j * C];
        zdft<T, R, true>(x);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          TS r0 = (TS)x[j].x, r1 = (TS)x[j].y;
          if (MODE != ZIX_FIELDS && MODE != ZIX_GRAD) {
            r0 = (TS)((T)a[j].a - x[j].x);
            r1 = (TS)((T)a[j].b - x[j].y);
          }
          stpair(out + o + j * step * xs, r0, r1, vec, two);
        }
      });
      return;
    }
    // The potential: levels z (but the block's first, the one below's) and z + 1
    // are stored, and the interfaces at both get their difference.
    if (pot) {
      const unsigned group = (C == 32 ? ~0u : (1u << C) - 1) << ((threadIdx.x & 31) & ~(C - 1));
      z_last_inv<T, C>(p, b0, RY, [&](auto rc, int row, int n, int step, const cplx<T>* q) {
        constexpr int R = decltype(rc)::value;
        if (row >= rows) return;  // the same for the lanes of a group
        const int o = (n * ny + y0 + row) * nz + z, wo = (n * ny + y0 + row) * (nz + 1) + z;
        const bool la = c > 0 && on, lb = two;
        TS a[R], b[R], fa[R], fb[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
          a[j] = la ? w_in[wo + j * step * ws] : (TS)0;
          b[j] = lb ? w_in[wo + j * step * ws + 1] : (TS)0;
          if (MODE == ZIX_REFINE) {
            fa[j] = la ? phi_out[o + j * step * xs] : (TS)0;
            fb[j] = lb ? phi_out[o + j * step * xs + 1] : (TS)0;
          }
        }
        if (MODE == ZIX_STAGE) {
#pragma unroll
          for (int j = 0; j < R; ++j) {
            const TS* t = bh + wo + j * step * ws;
            if (la) a[j] = (TS)zstage1<T>((T)a[j], sd, (T)t[0]);
            if (lb) b[j] = (TS)zstage1<T>((T)b[j], sd, (T)t[1]);
          }
        }
        cplx<T> x[R];
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = q[j * C];
        zdft<T, R, true>(x);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const T below = __shfl_up_sync(group, x[j].y, 1, C);
          const int k = j * step * xs, kw = j * step * ws;
          if (la) {
            w_out[wo + kw] = (TS)((T)a[j] - (x[j].x - below) * idz);
            phi_out[o + k] = (TS)(MODE == ZIX_REFINE ? (T)fa[j] + x[j].x : x[j].x);
          }
          if (lb) {  // no correction at the surface
            const T d = one ? (x[j].y - x[j].x) * idz : (T)0;
            w_out[wo + kw + 1] = (TS)((T)b[j] - d);
            phi_out[o + k + 1] = (TS)(MODE == ZIX_REFINE ? (T)fb[j] + x[j].y : x[j].y);
          }
        }
        // the lid level keeps the input's value (stages: with its buoyancy)
        if ((MODE == ZIX_STAGE || w_out != w_in) && ((la && z == nz - 1) || (lb && z + 2 == nz))) {
          for (int j = 0; j < R; ++j) {
            const int top = wo + j * step * ws + (nz - z);
            TS t = w_in[top];
            if (MODE == ZIX_STAGE) t = (TS)zstage1<T>((T)t, sd, (T)bh[top]);
            w_out[top] = t;
          }
        }
      });
      return;
    }
    z_last_inv<T, C>(p, b0, RY, [&](auto rc, int row, int n, int step, const cplx<T>* line) {
      constexpr int R = decltype(rc)::value;
      if (!on || row >= rows) return;
      const int o = (n * ny + y0 + row) * (nz + 1) + z;
      TS a[R], b[R];
      if (MODE != ZIX_GRAD) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          a[j] = w_in[o + j * step * ws];
          b[j] = w_in[o + j * step * ws + 1];
        }
        if (MODE == ZIX_STAGE) {
#pragma unroll
          for (int j = 0; j < R; ++j) {
            const TS* q = bh + o + j * step * ws;
            a[j] = (TS)zstage1<T>((T)a[j], sd, (T)q[0]);
            b[j] = (TS)zstage1<T>((T)b[j], sd, (T)q[1]);
          }
        }
      }
      cplx<T> x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = line[j * C];
      zdft<T, R, true>(x);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        TS* q = w_out + o + j * step * ws;
        if (MODE == ZIX_GRAD) {
          q[0] = (TS)x[j].x;
          if (two) q[1] = (TS)x[j].y;
          if (z + 2 >= nz) q[two ? 2 : 1] = (TS)0;
        } else {
          q[0] = (TS)((T)a[j] - x[j].x);
          if (two) q[1] = (TS)((T)b[j] - x[j].y);
        }
      }
      // the lid level keeps the input's value (stages: with its buoyancy)
      if (MODE != ZIX_GRAD && z + 2 >= nz && (MODE == ZIX_STAGE || w_out != w_in)) {
        for (int j = 0; j < R; ++j) {
          const int top = o + j * step * ws + (two ? 2 : 1);
          TS t = w_in[top];
          if (MODE == ZIX_STAGE) t = (TS)zstage1<T>((T)t, sd, (T)bh[top]);
          w_out[top] = t;
        }
      }
    });
}

// ---- y lines ---------------------------------------------------------------------
// One level of one kx per column; rows of a CTA are consecutive kx.

// rows of a spectrum at one level into a line's first forward pass
template <class T, int C>
__device__ __forceinline__ void zy_first(const ZPlan& p, const GridK& g, cplx<T>* buf, int RY,
                                         int rows, int k0, int z, const cplx<T>* src) {
  const bool on = z < g.nz;
  z_first_fwd<T, C>(p, buf, RY, [&](auto rc, int row, int c, int n, int step, cplx<T>* v) {
    constexpr int R = decltype(rc)::value;
    if (!on || row >= rows) return;
    const int o = ((k0 + row) * g.ny + n) * g.nz + z;
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = src[o + j * step * g.nz];
  });
}

// a line's last inverse pass into the rows of a spectrum
template <class T, int C>
__device__ __forceinline__ void zy_last(const ZPlan& p, const GridK& g, const cplx<T>* buf,
                                        int RY, int rows, int k0, int z, cplx<T>* dst) {
  const bool on = z < g.nz;
  z_last_inv<T, C>(p, buf, RY, [&](auto rc, int row, int n, int step, const cplx<T>* q) {
    constexpr int R = decltype(rc)::value;
    if (!on || row >= rows) return;
    cplx<T> x[R];
#pragma unroll
    for (int j = 0; j < R; ++j) x[j] = q[j * C];
    zdft<T, R, true>(x);
    const int o = ((k0 + row) * g.ny + n) * g.nz + z;
#pragma unroll
    for (int j = 0; j < R; ++j) dst[o + j * step * g.nz] = x[j];
  });
}

// Forward y of one field (ZFY_FIELDS).
template <class T>
__global__ void __launch_bounds__(kZThreads, sizeof(T) == 4 ? 3 : 2) k_zfy(
    const __grid_constant__ ZPlan p, GridK g, int RY, const cplx<T>* X0,
    const cplx<T>* __restrict__ tw, cplx<T>* out0) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int C = zy_cols<T>();
  constexpr int LC = zlog2(C);
  cplx<T>* b0 = reinterpret_cast<cplx<T>*>(smem_dyn);
  const int ny = g.ny, nz = g.nz;
  const int k0 = blockIdx.y * RY;
  const int z = blockIdx.x * C + (threadIdx.x & (C - 1));
  const bool on = z < nz;
  const int rows = min(RY, g.nxh - k0);
  zy_first<T, C>(p, g, b0, RY, rows, k0, z, X0);
  __syncthreads();
#pragma unroll 1
  for (int i = 1; i + 1 < p.np; ++i) {
    z_mid_pass<T, C, false>(p, i, b0, RY, tw);
    __syncthreads();
  }
  z_pair(p.r[p.np - 1], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int tot = RY * p.Q * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      int t = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dnb[p.np - 1].div(t);
        t -= row * p.Q;
      }
      if (!on || row >= rows) continue;
      cplx<T>* o = out0 + ((k0 + row) * ny + t) * nz + z;
      cplx<T> a[R];
      z_last_bfly<T, R, C>(p, b0 + (size_t)row * p.NP * C + (e & (C - 1)), t, tw, a);
#pragma unroll
      for (int j = 0; j < R; ++j) o[j * p.Q * nz] = a[j];
    }
  });
}

// Forward y of two fields, both lines in shared memory: ZFY_DIV, ZFY_RESID (the sum rounded to TO once) and ZFY_HELM (multipliers that mix the
// two, then both lines back).
template <class T, class TO, int MODE, int C>
__global__ void __launch_bounds__(kZThreads, sizeof(T) == 4 ? 3 : 2) k_zfy2(
    const __grid_constant__ ZPlan p, GridK g, int RY, const cplx<T>* X0, const cplx<T>* X1,
    double s_, const T* __restrict__ ky, const double* __restrict__ kxd,
    const double* __restrict__ kyd, const cplx<T>* __restrict__ tw, cplx<TO>* out0,
    cplx<T>* out1) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int LC = zlog2(C);
  cplx<T>* b0 = reinterpret_cast<cplx<T>*>(smem_dyn);
  cplx<T>* b1 = b0 + (size_t)RY * p.NP * C;
  const int ny = g.ny, nz = g.nz;
  const int k0 = blockIdx.y * RY;
  const int z = blockIdx.x * C + (threadIdx.x & (C - 1));
  const bool on = z < nz;
  const int rows = min(RY, g.nxh - k0);
#pragma unroll
  for (int f = 0; f < 2; ++f)
    zy_first<T, C>(p, g, f ? b1 : b0, RY, rows, k0, z, f ? X1 : X0);
  __syncthreads();
#pragma unroll 1
  for (int i = 1; i + 1 < p.np; ++i) {
#pragma unroll
    for (int f = 0; f < 2; ++f) z_mid_pass<T, C, false>(p, i, f ? b1 : b0, RY, tw);
    __syncthreads();
  }
  z_pair(p.r[p.np - 1], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int tot = RY * p.Q * C;
    for (int e = ztid(); e < tot; e += blockDim.x) {
      int t = e >> LC, row = 0;
      if (RY > 1) {
        row = p.dnb[p.np - 1].div(t);
        t -= row * p.Q;
      }
      if (!on || row >= rows) continue;
      const size_t lo = (size_t)row * p.NP * C + (e & (C - 1));
      const int kx = k0 + row;
      cplx<T> a[R], b[R];
      z_last_bfly<T, R, C>(p, b0 + lo, t, tw, a);
      z_last_bfly<T, R, C>(p, b1 + lo, t, tw, b);
      if constexpr (MODE == ZFY_HELM) {
        const double Kx = kxd[kx];
        const bool nyqx = kx == g.nx / 2;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int k = t + p.Q * j;
          const double Ky = kyd[k];
          const double K2 = Kx * Kx + Ky * Ky;
          const double q = K2 > 0 ? s_ / K2 : 0.0;
          const T mxx = (T)(q * Kx * Kx), myy = (T)(q * Ky * Ky);
          const T mxy = nyqx != (2 * k == ny) ? (T)0 : (T)(q * Kx * Ky);
          const cplx<T> U = a[j], V = b[j];
          a[j] = mk<T>(mxx * U.x + mxy * V.x, mxx * U.y + mxy * V.y);
          b[j] = mk<T>(mxy * U.x + myy * V.x, mxy * U.y + myy * V.y);
        }
        z_first_bfly_inv<T, R, C>(p, b0 + lo, t, tw, a);
        z_first_bfly_inv<T, R, C>(p, b1 + lo, t, tw, b);
      } else {
        cplx<TO>* o = out0 + (kx * ny + t) * nz + z;
        const int st = p.Q * nz;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int k = t + p.Q * j;
          cplx<T> d = add(a[j], ik(__ldg(ky + k), b[j]));
          if (MODE == ZFY_RESID && (2 * k == ny || 2 * kx == g.nx)) d = mk<T>((T)0, (T)0);
          o[j * st] = mk<TO>((TO)d.x, (TO)d.y);
        }
      }
    }
  });
  if constexpr (MODE == ZFY_HELM) {
    __syncthreads();
#pragma unroll 1
    for (int i = p.np - 2; i >= 1; --i) {
#pragma unroll
      for (int f = 0; f < 2; ++f) z_mid_pass<T, C, true>(p, i, f ? b1 : b0, RY, tw);
      __syncthreads();
    }
    zy_last<T, C>(p, g, b0, RY, rows, k0, z, out0);
    zy_last<T, C>(p, g, b1, RY, rows, k0, z, out1);
  }
}

// inverse y: out0 = F^-1(scale in), out1 (GRAD) = F^-1(i ky' scale in)
template <class T, bool GRAD>
__global__ void __launch_bounds__(kZThreads, sizeof(T) == 4 ? 3 : 2) k_ziy(
    const __grid_constant__ ZPlan p, GridK g, int RY, const cplx<T>* in, double scale,
    const T* __restrict__ ky, const cplx<T>* __restrict__ tw, cplx<T>* out0, cplx<T>* out1) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int C = zy_cols<T>();
  constexpr int LC = zlog2(C);
  cplx<T>* b0 = reinterpret_cast<cplx<T>*>(smem_dyn);
  const int ny = g.ny, nz = g.nz;
  const int k0 = blockIdx.y * RY;
  const int z = blockIdx.x * C + (threadIdx.x & (C - 1));
  const bool on = z < nz;
  const int rows = min(RY, g.nxh - k0);
  const T sc = (T)scale;
#pragma unroll 1
  for (int run = 0; run < (GRAD ? 2 : 1); ++run) {
    if (run) __syncthreads();
    z_pair(p.r[p.np - 1], [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int tot = RY * p.Q * C;
      for (int e = ztid(); e < tot; e += blockDim.x) {
        int t = e >> LC, row = 0;
        if (RY > 1) {
          row = p.dnb[p.np - 1].div(t);
          t -= row * p.Q;
        }
        if (!on || row >= rows) continue;
        const size_t lo = (size_t)row * p.NP * C + (e & (C - 1));
        const int o = ((k0 + row) * ny + t) * nz + z, st = p.Q * nz;
        cplx<T> a[R];
#pragma unroll
        for (int j = 0; j < R; ++j) a[j] = scl(in[o + j * st], sc);
        if (GRAD && run) {
#pragma unroll
          for (int j = 0; j < R; ++j) a[j] = ik(__ldg(ky + t + p.Q * j), a[j]);
        }
        z_first_bfly_inv<T, R, C>(p, b0 + lo, t, tw, a);
      }
    });
    __syncthreads();
#pragma unroll 1
    for (int i = p.np - 2; i >= 1; --i) {
      z_mid_pass<T, C, true>(p, i, b0, RY, tw);
      __syncthreads();
    }
    zy_last<T, C>(p, g, b0, RY, rows, k0, z, run ? out1 : out0);
  }
}

}  // namespace ob
