// Instances and launchers of the level-paired line transforms.  Compiled once
// per precision (-DOB_ZREAL=float -DOB_ZELEM=4, double and 8) and part: -DOB_ZPART=2, 4, 6, 8 the x
// kernels of lines whose last radix that is, -DOB_ZPART=0 the y kernels, the
// dispatch and (single precision) the line plans.
#include <algorithm>
#include <cstdlib>

#include "zfft.cuh"
#if OB_ZPART == 0
#include "zplane.cuh"
#endif

namespace ob {

namespace {

constexpr size_t kZSmemMax = 227 * 1024;
constexpr size_t kZSmemShare = 176 * 1024;
constexpr long kZFill = 2 * 148;  // CTAs below which lines are not batched

// Lines per CTA and threads: at least 128 threads' worth of radix-8
// butterflies, unless batching lines would leave the SMs short of CTAs.
struct Shape {
  int rows, threads;
  dim3 grid;
  size_t smem;
};
template <class T>
Shape shape(const ZPlan& p, int C, int nbuf, int lines, int chunks, int most) {
  Shape s;
  const int per = std::max(1, p.N * C / 8);
  int rows = std::max(1, 128 / per);
  while (rows > 1 && ((long)chunks * ((lines + rows - 1) / rows) < kZFill ||
                      (size_t)nbuf * rows * p.NP * C * 2 * sizeof(T) > kZSmemMax))
    --rows;
  s.rows = rows;
  s.threads = std::min(most, std::max(64, (rows * per + 31) / 32 * 32));
  s.grid = dim3(chunks, (lines + rows - 1) / rows);
  s.smem = (size_t)nbuf * rows * p.NP * C * 2 * sizeof(T);
  // Where the resident blocks' lines would take most of the SM's memory, one
  // block fewer leaves the first-level cache room for the rows' neighbouring
  // accesses (1024 points, single precision: forward y 456 -> 372 us): ask for
  // enough that it does not fit.
  const size_t resident = std::min<size_t>(65536 / ((sizeof(T) == 4 ? 80 : 128) * s.threads),
                                           kZSmemMax / s.smem);
  if (resident > 2 && resident * s.smem > kZSmemShare) s.smem = kZSmemMax / resident + 1024;
  return s;
}

template <class K>
cudaError_t attr(K k) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZSmemMax);
}

int div_up(int a, int b) { return (a + b - 1) / b; }

}  // namespace

using T = OB_ZREAL;
#define OB_ZWIDE (OB_ZELEM == 8)

#define OB_Z(call)                              \
  do {                                          \
    const cudaError_t e_ = (call);              \
    if (e_ != cudaSuccess) return e_;           \
  } while (0)

// x launchers of one last radix
template <class T, class TS, int RL>
cudaError_t zfx_last(int mode, const ZLine<T>& l, const GridK& g, const TS* u, const TS* v,
                     const TS* w, const TS* bh, double sdt, const double* rho,
                     const double* rhoh, cplx<T>* X0, cplx<T>* X1, cudaStream_t st);
template <class T, int RL>
cudaError_t zix_last(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* S1,
                     const cplx<T>* S2, const T* u, const T* v, const T* w, const T* bh,
                     double sdt, T* uo, T* vo, T* wo, T* phio, cudaStream_t st);
template <class T, int RL>
cudaError_t zx_init();

#if OB_ZPART > 0

template <class T, int RL>
cudaError_t zx_init() {
  OB_Z(attr(k_zfx<T, T, ZFX_DIV, RL>));
  OB_Z(attr(k_zfx<T, T, ZFX_STAGE, RL>));
  OB_Z(attr(k_zfx<T, T, ZFX_FIELDS, RL>));
  OB_Z(attr(k_zix<T, T, ZIX_CORRECT, RL>));
  OB_Z(attr(k_zix<T, T, ZIX_STAGE, RL>));
  OB_Z(attr(k_zix<T, T, ZIX_REFINE, RL>));
  OB_Z(attr(k_zix<T, T, ZIX_FIELDS, RL>));
  OB_Z(attr(k_zix<T, T, ZIX_GRAD, RL>));
  if constexpr (sizeof(T) == 8) OB_Z(attr(k_zfx<T, float, ZFX_DIV, RL>));
  return cudaSuccess;
}

template <class T, class TS, int RL>
cudaError_t zfx_last(int mode, const ZLine<T>& l, const GridK& g, const TS* u, const TS* v,
                     const TS* w, const TS* bh, double sdt, const double* rho,
                     const double* rhoh, cplx<T>* X0, cplx<T>* X1, cudaStream_t st) {
  constexpr int C = zx_pairs<T>();
  const int sets = mode == ZFX_FIELDS && !v ? 1 : 2;
  const Shape s = shape<T>(l.plan, C, 1, g.ny, sets * div_up(g.nz, 2 * C), zx_threads<T>());
  const bool pairs = zpairs<TS>(g.nz, u, v);
#define OB_ZFX(M)                                                                              \
  case M:                                                                                      \
    k_zfx<T, TS, M, RL><<<s.grid, s.threads, s.smem, st>>>(l.plan, g, s.rows, pairs, u, v, w, bh, \
                                                           sdt, rho, rhoh, l.k, l.tw, X0, X1); \
    break;
  if constexpr (sizeof(TS) != sizeof(T)) {
    switch (mode) { OB_ZFX(ZFX_DIV) default: return cudaErrorInvalidValue; }
  } else {
    switch (mode) {
      OB_ZFX(ZFX_DIV)
      OB_ZFX(ZFX_STAGE)
      OB_ZFX(ZFX_FIELDS)
      default: return cudaErrorInvalidValue;
    }
  }
#undef OB_ZFX
  return cudaGetLastError();
}

template <class T, int RL>
cudaError_t zix_last(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* S1,
                     const cplx<T>* S2, const T* u, const T* v, const T* w, const T* bh,
                     double sdt, T* uo, T* vo, T* wo, T* phio, cudaStream_t st) {
  constexpr int C = zx_pairs<T>();
  const int chunks = div_up(g.nz, 2 * C);
  const int blocks = mode == ZIX_FIELDS ? (S2 ? 2 : 1) * chunks
                     : mode != ZIX_GRAD && phio ? 2 * chunks + div_up(g.nz, 2 * C - 1)
                                                : 3 * chunks;
  const Shape s = shape<T>(l.plan, C, 1, g.ny, blocks, zx_threads<T>());
  const bool pairs = zpairs<T>(g.nz, u, v, uo, vo);
#define OB_ZIX(M)                                                                               \
  case M:                                                                                       \
    k_zix<T, T, M, RL><<<s.grid, s.threads, s.smem, st>>>(l.plan, g, s.rows, pairs, S1, S2, l.k, \
                                                          l.tw, u, v, w, bh, sdt, uo, vo, wo,   \
                                                          phio);                                \
    break;
  switch (mode) {
    OB_ZIX(ZIX_CORRECT)
    OB_ZIX(ZIX_STAGE)
    OB_ZIX(ZIX_REFINE)
    OB_ZIX(ZIX_FIELDS)
    OB_ZIX(ZIX_GRAD)
    default: return cudaErrorInvalidValue;
  }
#undef OB_ZIX
  return cudaGetLastError();
}

#define OB_ZFX_INST(TS)                                                                       \
  template cudaError_t zfx_last<T, TS, OB_ZPART>(                                             \
      int, const ZLine<T>&, const GridK&, const TS*, const TS*, const TS*, const TS*, double, \
      const double*, const double*, cplx<T>*, cplx<T>*, cudaStream_t);
OB_ZFX_INST(T)
#if OB_ZWIDE
OB_ZFX_INST(float)
#endif
template cudaError_t zix_last<T, OB_ZPART>(int, const ZLine<T>&, const GridK&, const cplx<T>*,
                                           const cplx<T>*, const T*, const T*, const T*,
                                           const T*, double, T*, T*, T*, T*, cudaStream_t);
template cudaError_t zx_init<T, OB_ZPART>();

#else  // OB_ZPART == 0

template <>
cudaError_t zfft_init<T>() {
  OB_Z((zx_init<T, 2>()));
  OB_Z((zx_init<T, 4>()));
  OB_Z((zx_init<T, 6>()));
  OB_Z((zx_init<T, 8>()));
  constexpr int C = zy_cols<T>();
  OB_Z(attr(k_zfy<T>));
  OB_Z(attr(k_zfy2<T, T, ZFY_DIV, C>));
  OB_Z(attr(k_zfy2<T, T, ZFY_HELM, C>));
  OB_Z(attr(k_zfy2<T, T, ZFY_DIV, C / 2>));
  OB_Z(attr(k_zfy2<T, T, ZFY_HELM, C / 2>));
  OB_Z(attr(k_ziy<T, true>));
  OB_Z(attr(k_ziy<T, false>));
  OB_Z(attr(k_zplane<T, false>));
  OB_Z(attr(k_zplane<T, true>));
#if OB_ZWIDE
  OB_Z(attr(k_zfy2<T, float, ZFY_RESID, C>));
  OB_Z(attr(k_zfy2<T, float, ZFY_RESID, C / 2>));
#endif
  return cudaSuccess;
}

#define OB_ZLASTS(CALL)                            \
  switch (l.plan.r[l.plan.np - 1]) {               \
    case 2: return CALL(2);                        \
    case 4: return CALL(4);                        \
    case 6: return CALL(6);                        \
    case 8: return CALL(8);                        \
  }                                                \
  return cudaErrorInvalidValue;

template <class T, class TS>
cudaError_t zfx(int mode, const ZLine<T>& l, const GridK& g, const TS* u, const TS* v,
                const TS* w, const TS* bh, double sdt, const double* rho, const double* rhoh,
                cplx<T>* X0, cplx<T>* X1, cudaStream_t st) {
#define OB_CALL(R) \
  zfx_last<T, TS, R>(mode, l, g, u, v, w, bh, sdt, rho, rhoh, X0, X1, st)
  OB_ZLASTS(OB_CALL)
#undef OB_CALL
}

template <class T>
cudaError_t zix(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* S1,
                const cplx<T>* S2, const T* u, const T* v, const T* w, const T* bh, double sdt,
                T* uo, T* vo, T* wo, T* phio, cudaStream_t st) {
#define OB_CALL(R) \
  zix_last<T, R>(mode, l, g, S1, S2, u, v, w, bh, sdt, uo, vo, wo, phio, st)
  OB_ZLASTS(OB_CALL)
#undef OB_CALL
}

// two lines per column: full columns where two CTAs per SM hold them
template <class T, class TO, int MODE>
cudaError_t zfy2(const ZLine<T>& l, const GridK& g, const cplx<T>* X0, const cplx<T>* X1,
                 double sc, const double* kxd, const double* kyd,
                 cplx<TO>* out0, cplx<T>* out1, cudaStream_t st) {
  constexpr int C = zy_cols<T>();
  if (2ull * l.plan.NP * C * 2 * sizeof(T) <= kZSmemMax / 2) {
    const Shape s = shape<T>(l.plan, C, 2, g.nxh, div_up(g.nz, C), kZThreads);
    k_zfy2<T, TO, MODE, C><<<s.grid, s.threads, s.smem, st>>>(
        l.plan, g, s.rows, X0, X1, sc, l.k, kxd, kyd, l.tw, out0, out1);
  } else {
    const Shape s = shape<T>(l.plan, C / 2, 2, g.nxh, div_up(g.nz, C / 2), kZThreads);
    k_zfy2<T, TO, MODE, C / 2><<<s.grid, s.threads, s.smem, st>>>(
        l.plan, g, s.rows, X0, X1, sc, l.k, kxd, kyd, l.tw, out0, out1);
  }
  return cudaGetLastError();
}

template <class T, class TO>
cudaError_t zfy(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* X0,
                const cplx<T>* X1, double sc, const double* kxd,
                const double* kyd, cplx<TO>* out0, cplx<T>* out1, cudaStream_t st) {
  if constexpr (sizeof(TO) != sizeof(T)) {
    if (mode != ZFY_RESID) return cudaErrorInvalidValue;
    return zfy2<T, TO, ZFY_RESID>(l, g, X0, X1, sc, kxd, kyd, out0, out1, st);
  } else {
    if (mode == ZFY_DIV)
      return zfy2<T, TO, ZFY_DIV>(l, g, X0, X1, sc, kxd, kyd, out0, out1, st);
    if (mode == ZFY_HELM)
      return zfy2<T, TO, ZFY_HELM>(l, g, X0, X1, sc, kxd, kyd, out0, out1, st);
    if (mode != ZFY_FIELDS) return cudaErrorInvalidValue;
    constexpr int C = zy_cols<T>();
    const Shape s = shape<T>(l.plan, C, 1, g.nxh, div_up(g.nz, C), kZThreads);
    k_zfy<T><<<s.grid, s.threads, s.smem, st>>>(l.plan, g, s.rows, X0, l.tw, out0);
    return cudaGetLastError();
  }
}

template <class T>
cudaError_t ziy(bool grad, const ZLine<T>& l, const GridK& g, const cplx<T>* in, double scale,
                cplx<T>* out0, cplx<T>* out1, cudaStream_t st) {
  constexpr int C = zy_cols<T>();
  const Shape s = shape<T>(l.plan, C, 1, g.nxh, div_up(g.nz, C), kZThreads);
  if (grad)
    k_ziy<T, true><<<s.grid, s.threads, s.smem, st>>>(l.plan, g, s.rows, in, scale, l.k, l.tw,
                                                      out0, out1);
  else
    k_ziy<T, false><<<s.grid, s.threads, s.smem, st>>>(l.plan, g, s.rows, in, scale, l.k, l.tw,
                                                       out0, out1);
  return cudaGetLastError();
}

template <>
int zplane_group<T>(const ZPlan& p, int nz) {
  const int C = zy_cols<T>(), nch = div_up(nz, C);
  int best = 0;
  for (int q = 1; q <= nch; ++q)
    if (zplane_layout<T>(p.NP, nz, q).total <= kZSmemMax) best = q;
  // groups of even size: as few as the largest one gives
  return best ? div_up(nch, div_up(nch, best)) : 0;
}

template <>
cudaError_t zplane<T>(const ZLine<T>& l, const GridK& g, const ThomasK& t, const ZSolve& s,
                      bool fwd, const cplx<T>* X0, const cplx<T>* X1, cplx<T>* out0, cplx<T>* out1,
                      const ZLog<T>& log, cudaStream_t st) {
  const int group = zplane_group<T>(l.plan, g.nz);
  if (!group) return cudaErrorInvalidValue;
  const size_t smem = zplane_layout<T>(l.plan.NP, g.nz, group).total;
  const int per = l.plan.N * div_up(g.nz, zy_cols<T>()) * zy_cols<T>() / 8;
  // a warp more than the columns fill, for the zero mode, where that costs none
  const int threads = std::min(kZPlaneThreads,
                               std::max({128, div_up(per, 64) * 64, div_up(g.ny, 32) * 32 + 32}));
  if (log.diag && !fwd) return cudaErrorInvalidValue;
  if (log.diag)
    k_zplane<T, true><<<g.nxh, threads, smem, st>>>(l.plan, g, group, fwd, X0, X1, l.k, l.tw, t,
                                                    s.inv, s.dpd, s.lw, out0, out1, log);
  else
    k_zplane<T, false><<<g.nxh, threads, smem, st>>>(l.plan, g, group, fwd, X0, X1, l.k, l.tw, t,
                                                     s.inv, s.dpd, s.lw, out0, out1, ZNoLog{});
  return cudaGetLastError();
}

#if OB_ZWIDE
cudaError_t zplane_inv(const GridK& g, const ThomasK& t, double* inv, cudaStream_t st) {
  k_zinv<<<div_up(g.nxh * g.ny, 128), 128, 0, st>>>(g, t, inv);
  return cudaGetLastError();
}
#endif

#define OB_ZFX_INST(TS)                                                                      \
  template cudaError_t zfx<T, TS>(int, const ZLine<T>&, const GridK&, const TS*, const TS*,  \
                                  const TS*, const TS*, double, const double*, const double*, \
                                  cplx<T>*, cplx<T>*, cudaStream_t);
#define OB_ZFY_INST(TO)                                                                      \
  template cudaError_t zfy<T, TO>(int, const ZLine<T>&, const GridK&, const cplx<T>*,        \
                                  const cplx<T>*, double, const double*,                     \
                                  const double*, cplx<TO>*, cplx<T>*, cudaStream_t);
OB_ZFX_INST(T)
OB_ZFY_INST(T)
#if OB_ZWIDE
OB_ZFX_INST(float)
OB_ZFY_INST(float)
#else
// Line plans.  Passes are as few as the radices allow (each one is a trip
// through shared memory and a barrier); among equals the radices next to
// global memory stay near 8 (the last one near 4 in double), which keeps a
// thread's loads and its two butterflies in registers, and an adjacent pass of
// 4, 8 or odd radix reads and writes shared memory without bank conflicts.
bool zplan_make(int N, int elem, ZPlan* out) {
  if (N < 4 || (N & 1)) return false;
  static const int edge[] = {8, 4, 9, 10, 6, 5, 3, 2};
  static const int mid[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
  static const int last[] = {8, 6, 4, 2};
  int best[4] = {0, 0, 0, 0}, bnp = 99;
  double bcost = 1e30;
  auto consider = [&](int np, const int* r) {
    // shared-memory trips, then butterflies of uneven or wide radix
    double c = 100.0 * np;
    for (int i = 0; i < np; ++i)
      c += std::abs(r[i] - (i == np - 1 && elem == 8 ? 4 : 8)) * (i == 0 || i == np - 1 ? 2.0 : 1.0);
    if (r[0] != 8 && r[0] != 4 && !(r[0] & 1)) c += 8;
    if (r[0] == 10) c += 4;
    if (c < bcost) {
      bcost = c;
      bnp = np;
      for (int i = 0; i < 4; ++i) best[i] = i < np ? r[i] : 1;
    }
  };
  for (int a : edge)
    for (int z : last) {
      if (N % (a * z)) continue;
      const int m = N / (a * z);
      int r[4];
      if (m == 1) {
        r[0] = a; r[1] = z;
        consider(2, r);
        continue;
      }
      for (int b : mid) {
        if (m % b) continue;
        if (m == b) {
          r[0] = a; r[1] = b; r[2] = z;
          consider(3, r);
          continue;
        }
        for (int c : mid)
          if (m == b * c) {
            r[0] = a; r[1] = b; r[2] = c; r[3] = z;
            consider(4, r);
          }
      }
    }
  if (bnp > 4) return false;
  ZPlan p{};
  p.N = N;
  p.np = bnp;
  int S = 1;
  for (int i = 0; i < 4; ++i) {
    p.r[i] = best[i];
    p.S[i] = S;
    if (i < bnp) {
      p.nb[i] = N / best[i];
      S *= best[i];
    } else {
      p.nb[i] = 1;
    }
    p.dS[i] = FastDiv((unsigned)p.S[i]);
    p.dnb[i] = FastDiv((unsigned)p.nb[i]);
    p.dr[i] = FastDiv((unsigned)p.r[i]);
  }
  p.Q = N / best[bnp - 1];
  p.ns = (p.Q + 1) / 2;
  p.dns = FastDiv((unsigned)p.ns);
  p.sh = 31;
  for (int s = 1; s <= 3; ++s)
    if (best[0] == (1 << s)) p.sh = s;
  p.NP = N + (N >> p.sh);
  // one line of every column (the y kernels that hold two have half as many)
  const size_t cols = elem == 4 ? 8 : 4;
  if (p.NP * cols * 2 * elem > kZSmemMax) return false;
  *out = p;
  return true;
}

void zplan_twiddles(const ZPlan& p, int* t) {
  for (int i = 0; i < p.N; ++i) t[i] = 0;
  for (int i = 1; i < p.np; ++i)
    for (int j = 1; j < p.r[i]; ++j)
      for (int k = 0; k < p.S[i]; ++k)
        t[p.S[i] - 1 + (j - 1) * p.S[i] + k] = j * k * (p.N / (p.S[i] * p.r[i]));
}
#endif  // OB_ZWIDE
template cudaError_t zix<T>(int, const ZLine<T>&, const GridK&, const cplx<T>*, const cplx<T>*,
                            const T*, const T*, const T*, const T*, double, T*, T*, T*, T*,
                            cudaStream_t);
template cudaError_t ziy<T>(bool, const ZLine<T>&, const GridK&, const cplx<T>*, double,
                            cplx<T>*, cplx<T>*, cudaStream_t);

#endif  // OB_ZPART

}  // namespace ob
