// Host interface of the level-paired line transforms (zfft.cuh): line plans and
// launchers, compiled apart from the C ABI (zfft.cu, once per precision).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace ob {

// A line's factorisation N = r[0] r[1] .. r[np-1].  Position of the digit
// vector (j0, j1, ..): j0 + S[1] j1 + S[2] j2 + ..; it holds input row
// n = j_last + r_last (j_prev + ..) before a forward transform and wavenumber
// j0 + S[1] j1 + .. after it.
struct ZPlan {
  int N, np, Q;     // Q = N / r[np-1]: stride of the last forward pass
  int r[4], S[4];   // radix and stride of each forward pass
  int nb[4];        // butterflies per line N / r[i]
  int sh, NP;       // pad shift, padded length
  int ns;           // butterfly pairs (t, Q - t) of the last forward pass
  FastDiv dS[4], dnb[4], dr[4], dns;
};

// The plan of an even line of N points with elements of `elem` bytes (4 or 8);
// false where N has no factorisation in the kernels' radices or a line of every
// column exceeds shared memory.
bool zplan_make(int N, int elem, ZPlan* out);

// The index into W_N^t of every entry of the line's pass twiddles (N entries).
void zplan_twiddles(const ZPlan& p, int* t);

// Whether the level pairs of a call's fields move as one access each: an even level
// count, so that every column starts on a pair, and every field on a multiple of the
// pair's size.  A caller's field need not: a view into a larger buffer starts on any
// element, and goes level by level.
template <class TS, class... P>
inline bool zpairs(int nz, const P*... fields) {
  return !(nz & 1) &&
         (... && (reinterpret_cast<std::uintptr_t>(fields) % (2 * sizeof(TS)) == 0));
}

// One direction's lines: plan and device tables.
template <class T>
struct ZLine {
  ZPlan plan;
  const T* k;          // wavenumbers, the Nyquist entry zeroed
  const cplx<T>* tw;   // pass twiddles (zplan_twiddles)
};

// forward x modes
#define ZFX_DIV 0     // X0 = i kx' F(rho u) + F(D w), X1 = F(rho v)
#define ZFX_STAGE 1   // the same of w + sdt b_half
#define ZFX_FIELDS 2  // X0 = F(u), X1 = F(v) (v null: X0 alone)
// inverse x modes
#define ZIX_CORRECT 0  // u, v, w -= grad phi; phi stored unless null
#define ZIX_STAGE 1    // out = (u, v, w + sdt b_half) - grad phi
#define ZIX_REFINE 2   // ZIX_CORRECT with phi += the line
#define ZIX_FIELDS 3   // uo = F^-1(S1), vo = F^-1(S2) (S2 null: uo alone)
#define ZIX_GRAD 4     // uo, vo, wo = the gradient (wo on nz + 1 levels, 0 at the ends)
// forward y modes
#define ZFY_DIV 0     // out0 = F(X0) + i ky' F(X1)
#define ZFY_RESID 1   // ZFY_DIV, zero on the Nyquist rows, rounded to TO
#define ZFY_FIELDS 2  // out0 = F(X0)
#define ZFY_HELM 3    // forward, the damper's multipliers (times s), and back

// Raises the kernels' shared-memory limits on the current device.
template <class T>
cudaError_t zfft_init();

template <class T, class TS>
cudaError_t zfx(int mode, const ZLine<T>& l, const GridK& g, const TS* u, const TS* v,
                const TS* w, const TS* bh, double sdt, const double* rho, const double* rhoh,
                cplx<T>* X0, cplx<T>* X1, cudaStream_t st);
template <class T>
cudaError_t zix(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* S1,
                const cplx<T>* S2, const T* u, const T* v, const T* w, const T* bh, double sdt,
                T* uo, T* vo, T* wo, T* phio, cudaStream_t st);
template <class T, class TO>
cudaError_t zfy(int mode, const ZLine<T>& l, const GridK& g, const cplx<T>* X0,
                const cplx<T>* X1, double s, const double* kxd,
                const double* kyd, cplx<TO>* out0, cplx<T>* out1, cudaStream_t st);
template <class T>
cudaError_t ziy(bool grad, const ZLine<T>& l, const GridK& g, const cplx<T>* in, double scale,
                cplx<T>* out0, cplx<T>* out1, cudaStream_t st);

// One kx plane per block (zplane.cuh): forward y, the vertical solve, inverse y.
// X1 null: the source is F(X0) alone; fwd false: X0 is the source's spectrum.
// out1 = F^-1(i ky' phi^), null: out0 = phi~ alone.
struct ZSolve {
  const double* inv;          // reciprocal pivots (nx / 2 + 1, nz, ny)
  cplx<double>* dpd;          // scratch of that shape, single precision only
  const unsigned char* lw;    // per 32 columns: long waves (single precision)
};
// Where a solve logs its residuals; diag null: it does not.
template <class T>
struct ZLog {
  double* diag;
  int slot_c, slot_d;   // compatibility residual; sum of |L phi^ - d^|^2, added to
  cplx<T>* src;         // scratch of the source's size, (nx / 2 + 1, ny, nz)
};
// level chunks per group of the plane's scratch; 0: the plane does not fit
template <class T>
int zplane_group(const ZPlan& p, int nz);
template <class T>
cudaError_t zplane(const ZLine<T>& l, const GridK& g, const ThomasK& t, const ZSolve& s,
                   bool fwd, const cplx<T>* X0, const cplx<T>* X1, cplx<T>* out0, cplx<T>* out1,
                   const ZLog<T>& log, cudaStream_t st);
cudaError_t zplane_inv(const GridK& g, const ThomasK& t, double* inv, cudaStream_t st);

}  // namespace ob
