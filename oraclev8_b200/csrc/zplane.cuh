// One kx plane's y transforms, vertical solve and inverse y transforms in one
// block, for planes (ny x nz) that fit shared memory.
//
// Separate launches write and read the plane's spectrum twice and, at the grids
// where a plane fits, each takes longer to start and drain than to run; the
// batched solve alone is a serial chain of divisions.  Here the plane stays in
// shared memory from the forward transform's first pass to the inverse's last:
//   forward lines of X0 in the plane, of X1 in a scratch of a few level chunks;
//   d^ = F(X0) + i ky' F(X1) back into the plane, natural wavenumber order;
//   one thread per column sweeps up and down in double with the plan's reciprocal
//   pivots (k_zinv), the reference's operation order without its divisions;
//   i ky' phi^ through the scratch into out1, phi^ in the plane into out0.
// What bounds it: the latency of its phases in one block per SM (barriers, the
// sweep's chain of dependent operations per level each way).  Measured, the three
// launches against this one (us): 128 x 128 x 32 double 44.6 -> 27; 96 x 96 x 32
// single 48 -> 23, 250 x 162 x 45 single 70 -> 39 (with the long waves' double
// sweep, which the separate solve runs beside the others).  Planes that need a
// second wave of blocks mostly lose: 320 x 320 x 32 double 91 -> 157.  A plan that
// is not tuned takes this form for grids of one wave; the autotuner times both.
#pragma once
#include "zfft.cuh"

namespace ob {

// Reciprocal pivots of the columns (kx, ky): inv[(kx nz + k) ny + ky], the
// forward elimination of poisson.py:286-332.
static __global__ void k_zinv(GridK g, ThomasK t, double* __restrict__ inv) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.nxh * g.ny) return;
  const int kx = col / g.ny, ky = col - kx * g.ny;
  double* o = inv + (size_t)kx * g.nz * g.ny + ky;
  const double a = t.kx[kx], b = t.ky[ky];
  const double ksq = arn(mrn(a, a), mrn(b, b));
  double cp = 0.0;
  for (int k = 0; k < g.nz; ++k) {
    const double d = srn(t.negs[k], mrn(ksq, t.rho[k]));
    // the zero mode (column 0) has its own reduced system
    const double r = col ? rcprn(k ? srn(d, mrn(t.a[k], cp)) : d) : 0.0;
    o[(size_t)k * g.ny] = r;
    cp = mrn(t.c[k], r);
  }
}

// Sweep of one column in double: values of type T at col[k] (k < nz), reciprocal
// pivots at inv[k ny]; DP: the eliminated values wait for the way back in dp,
// else in the column, rounded to T.  Pivots (and dp on the way back) are loaded a
// batch ahead of the chain that uses them; first: the pivots of levels
// 0 .. kZBatch - 1, loaded before the block's barrier.  LOG: returns the sum of
// |L phi^ - d^|^2 over the levels (poisson.py:263-268), of the column's solution
// as it is found (DP and double: before its last rounding) and its source in r.
constexpr int kZBatch = 8;
// One column's source, as the plane's solve found it, and what L needs of it.
template <class T>
struct ZResid {
  const cplx<T>* d;    // nz levels
  const double *rho, *rhoh;
  double ksq, dz2;
};
__device__ __forceinline__ void z_pivots(double* v, const double* __restrict__ inv, int k0,
                                         int nz, int ny) {
#pragma unroll
  for (int j = 0; j < kZBatch; ++j)
    v[j] = (k0 + j >= 0 && k0 + j < nz) ? __ldg(inv + (size_t)(k0 + j) * ny) : 0.0;
}
template <class T, bool DP, bool LOG>
__device__ __forceinline__ double z_sweep(cplx<T>* col, int nz, int ny,
                                          const double* __restrict__ inv, const double* a,
                                          const double* c, double scale, cplx<double>* dp,
                                          const double* first, const ZResid<T>& r) {
  double cur[kZBatch], nxt[kZBatch];
  double pr = 0.0, pi = 0.0;
#pragma unroll
  for (int j = 0; j < kZBatch; ++j) nxt[j] = first[j];
#pragma unroll 1
  for (int k0 = 0; k0 < nz; k0 += kZBatch) {
#pragma unroll
    for (int j = 0; j < kZBatch; ++j) cur[j] = nxt[j];
    z_pivots(nxt, inv, k0 + kZBatch, nz, ny);
    const int n = min(kZBatch, nz - k0);
#pragma unroll
    for (int j = 0; j < kZBatch; ++j) {
      if (j >= n) break;
      const int k = k0 + j;  // a[0] = 0
      const cplx<T> d = col[k];
      pr = mrn(srn((double)d.x, mrn(a[k], pr)), cur[j]);
      pi = mrn(srn((double)d.y, mrn(a[k], pi)), cur[j]);
      if (DP) dp[(size_t)k * ny] = mk<double>(pr, pi);
      else col[k] = mk<T>((T)pr, (T)pi);
    }
  }
  col[nz - 1] = mk<T>((T)(pr * scale), (T)(pi * scale));
  // residual: the level above and the flux through its top
  double acc = 0.0, ur = 0.0, ui = 0.0, fr = 0.0, fi = 0.0;
  auto as_found = [](double x) { return DP ? x : (double)(T)x; };
  auto row = [&](int k, double fur, double fui, double flr, double fli) {  // level k, (ur, ui)
    const cplx<T> d = r.d[k];
    const double q = r.ksq * r.rho[k];
    const double rr = (fur - flr) / r.dz2 - q * ur - (double)d.x;
    const double ri = (fui - fli) / r.dz2 - q * ui - (double)d.y;
    acc += rr * rr + ri * ri;
  };
  if (LOG) {
    ur = as_found(pr);
    ui = as_found(pi);
  }
  // batches downward from level nz - 2: levels k0 .. k0 - kZBatch + 1
  cplx<double> dc[DP ? kZBatch : 1], dn[DP ? kZBatch : 1];
  auto values = [&](int k0) {
    z_pivots(nxt, inv, k0 - kZBatch + 1, nz, ny);
    if (DP) {
#pragma unroll
      for (int j = 0; j < (DP ? kZBatch : 1); ++j) {
        const int k = k0 - j;
        if (k >= 0) dn[j] = dp[(size_t)k * ny];
      }
    }
  };
  values(nz - 2);
#pragma unroll 1
  for (int k0 = nz - 2; k0 >= 0; k0 -= kZBatch) {
#pragma unroll
    for (int j = 0; j < kZBatch; ++j) {
      cur[j] = nxt[kZBatch - 1 - j];
      if (DP) dc[DP ? j : 0] = dn[DP ? j : 0];
    }
    values(k0 - kZBatch);
    const int n = min(kZBatch, k0 + 1);
#pragma unroll
    for (int j = 0; j < kZBatch; ++j) {
      if (j >= n) break;
      const int k = k0 - j;
      const double cp = mrn(c[k], cur[j]);
      const cplx<double> d = DP ? dc[DP ? j : 0] : mk<double>((double)col[k].x, (double)col[k].y);
      pr = srn(d.x, mrn(cp, pr));
      pi = srn(d.y, mrn(cp, pi));
      col[k] = mk<T>((T)(pr * scale), (T)(pi * scale));
      if (LOG) {
        const double xr = as_found(pr), xi = as_found(pi);
        const double flr = r.rhoh[k + 1] * (ur - xr), fli = r.rhoh[k + 1] * (ui - xi);
        row(k + 1, fr, fi, flr, fli);
        fr = flr;
        fi = fli;
        ur = xr;
        ui = xi;
      }
    }
  }
  if (LOG) row(0, fr, fi, 0.0, 0.0);
  return acc;
}

// The zero mode (poisson.py:256, 316-325, 367-383) of one column, in double: the
// mean removed, the reduced system with phi(0, 0, 0) = 0.  w: 5 nz doubles, the
// last 3 nz the reduced system's a0, cp0, inv0.  LOG: returns the residual against
// the whole source less its mean (the zero mode of a real field is real), and the
// compatibility residual (poisson.py:233-236) in *compat.
template <class T, bool LOG>
__device__ double z_zero_mode(cplx<T>* col, int nz, double scale, double* w, const ZResid<T>& r,
                              double dz, double* compat) {
  const double *a0 = w + 2 * nz, *cp0 = w + 3 * nz, *inv0 = w + 4 * nz;
  double sr = 0, si = 0;
#pragma unroll 4
  for (int k = 0; k < nz; ++k) {
    sr = arn(sr, (double)col[k].x);
    si = arn(si, (double)col[k].y);
  }
  if (LOG) *compat = hypot(mrn(sr, dz), mrn(si, dz));
  const double mr = drn(sr, (double)nz), mi = drn(si, (double)nz);
  double pr = 0, pi = 0;
#pragma unroll 4
  for (int j = 0; j < nz - 1; ++j) {  // a0[0] = 0
    const double dr = srn((double)col[j + 1].x, mr), di = srn((double)col[j + 1].y, mi);
    pr = mrn(srn(dr, mrn(a0[j], pr)), inv0[j]);
    pi = mrn(srn(di, mrn(a0[j], pi)), inv0[j]);
    w[2 * j] = pr;
    w[2 * j + 1] = pi;
  }
  col[0] = mk<T>((T)0, (T)0);
  col[nz - 1] = mk<T>((T)(pr * scale), (T)(pi * scale));
  double above = pr, fu = 0.0, s1 = 0.0, s2 = 0.0;
  auto row = [&](int k, double fl) {  // of level k: its value above, the flux fl below it
    const double q = (fu - fl) / r.dz2 - (double)r.d[k].x;
    s1 += q;
    s2 += q * q;
    fu = fl;
  };
#pragma unroll 4
  for (int j = nz - 3; j >= 0; --j) {
    pr = srn(w[2 * j], mrn(cp0[j], pr));
    pi = srn(w[2 * j + 1], mrn(cp0[j], pi));
    col[j + 1] = mk<T>((T)(pr * scale), (T)(pi * scale));
    if (LOG) {
      row(j + 2, r.rhoh[j + 2] * (above - pr));
      above = pr;
    }
  }
  if (!LOG) return 0.0;
  row(1, r.rhoh[1] * above);
  row(0, 0.0);
  return s2 - s1 * s1 / nz;
}

constexpr int kZPlaneThreads = 512;

// a kernel that logs nothing takes no argument for it
struct ZNoLog {};
template <class T, bool LOG>
using ZLogArg = std::conditional_t<LOG, ZLog<T>, ZNoLog>;

// Shared memory of a plane block (bytes from the dynamic base): the plane's
// slots (every column of a wavenumber, their count made odd so the sweep's
// lanes fall on distinct banks), the scratch lines of `group` level chunks, the
// vertical operator's off-diagonals and the zero mode's values.
struct ZPlaneLayout {
  size_t scratch, a, c, zero, total;
  int st;  // elements between slots
};
template <class T>
__host__ __device__ inline ZPlaneLayout zplane_layout(int NP, int nz, int group) {
  auto al = [](size_t b) { return (b + 15) & ~size_t(15); };
  ZPlaneLayout L;
  const size_t ce = 2 * sizeof(T);
  const int C = zy_cols<T>();
  L.st = (nz + C - 1) / C * C | 1;
  L.scratch = al(NP * ce * L.st);
  L.a = L.scratch + al(NP * ce * C * group);
  L.c = L.a + al(nz * sizeof(double));
  L.zero = L.c + al(nz * sizeof(double));
  L.total = L.zero + al(5 * nz * sizeof(double));
  return L;
}

// grid = nx / 2 + 1 blocks.  X1 null: d^ = F(X0); fwd 0: X0 is d^ itself.  out1
// null: phi~ alone.  The outputs may be the inputs (a block reads its plane before
// it writes).  inv: reciprocal pivots.  Single precision: the columns of a block
// of 32 that lw flags (nearly singular, long waves) keep their eliminated values
// in double, in dpd.  LOG (with fwd): the residuals of this solution into log, the
// source kept in log.src until the sweep returns to it; the solution is the one an
// unlogged solve gives.
template <class T, bool LOG>
__global__ void __launch_bounds__(kZPlaneThreads, 1) k_zplane(
    const __grid_constant__ ZPlan p, GridK g, int group, int fwd, const cplx<T>* X0,
    const cplx<T>* X1, const T* __restrict__ ky, const cplx<T>* __restrict__ tw,
    const __grid_constant__ ThomasK t, const double* __restrict__ inv, cplx<double>* dpd,
    const unsigned char* __restrict__ lw, cplx<T>* out0, cplx<T>* out1, ZLogArg<T, LOG> log) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  constexpr int C = zy_cols<T>();
  constexpr int LC = zlog2(C);
  const int ny = g.ny, nz = g.nz, kx = blockIdx.x;
  const ZPlaneLayout L = zplane_layout<T>(p.NP, nz, group);
  cplx<T>* pl = reinterpret_cast<cplx<T>*>(smem_dyn);
  cplx<T>* sc = reinterpret_cast<cplx<T>*>(smem_dyn + L.scratch);
  double* ad = reinterpret_cast<double*>(smem_dyn + L.a);
  double* cd = reinterpret_cast<double*>(smem_dyn + L.c);
  const int st = L.st, srs = p.NP * C;
  const int nch = (nz + C - 1) / C;
  for (int k = threadIdx.x; k < nz; k += blockDim.x) {
    ad[k] = t.a[k];
    cd[k] = t.c[k];
  }
  double* zw = reinterpret_cast<double*>(smem_dyn + L.zero);
  if (kx == 0)
    for (int j = threadIdx.x; j < nz - 1; j += blockDim.x) {
      zw[2 * nz + j] = t.a0[j];
      zw[3 * nz + j] = t.cp0[j];
      zw[4 * nz + j] = t.inv0[j];
    }
  // both lines of every column at once where the scratch holds them
  const bool whole = group >= nch;
  // rows n, n + step, .. of a spectrum's plane, level chunk `row` past ch0
  auto rows = [&](const cplx<T>* src, int ch0) {
    return [=](auto rc, int row, int c, int n, int step, cplx<T>* v) {
      constexpr int R = decltype(rc)::value;
      const int z = (ch0 + row) * C + c;
      const cplx<T>* q = src + (kx * ny + n) * nz + z;
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = z < nz ? q[j * step * nz] : mk<T>((T)0, (T)0);
    };
  };
  auto store = [&](cplx<T>* dst, int ch0, int slot) {
    return [=](auto rc, int row, int n, int step, const cplx<T>* q) {
      constexpr int R = decltype(rc)::value;
      const int z = (ch0 + row) * C + (threadIdx.x & (C - 1));
      if (z >= nz) return;
      cplx<T> x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = q[j * slot];
      zdft<T, R, true>(x);
      const int o = (kx * ny + n) * nz + z;
#pragma unroll
      for (int j = 0; j < R; ++j) dst[o + j * step * nz] = x[j];
    };
  };

  if (!fwd) {
    for (int e = threadIdx.x; e < ny * nz; e += blockDim.x) {
      const int k = e / nz, z = e - k * nz;
      pl[zphys(p, k) * st + z] = X0[kx * ny * nz + e];
    }
    // columns past the last level are transformed with the others
    for (int e = threadIdx.x; e < ny * (nch * C - nz); e += blockDim.x) {
      const int k = e / (nch * C - nz), z = nz + e - k * (nch * C - nz);
      pl[zphys(p, k) * st + z] = mk<T>((T)0, (T)0);
    }
  } else {
    // forward lines of X0, in the plane
    z_first_fwd<T, C>(p, pl, nch, rows(X0, 0), st, C);
    if (whole && X1) z_first_fwd<T, C>(p, sc, nch, rows(X1, 0));
    __syncthreads();
#pragma unroll 1
    for (int i = 1; i + 1 < p.np; ++i) {
      z_mid_pass<T, C, false>(p, i, pl, nch, tw, st, C);
      if (whole && X1) z_mid_pass<T, C, false>(p, i, sc, nch, tw);
      __syncthreads();
    }
    // of X1, a group of chunks at a time, and both into d^
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += group) {
      const int n = min(group, nch - c0);
      if (X1 && !whole) {
        if (c0) __syncthreads();
        z_first_fwd<T, C>(p, sc, n, rows(X1, c0));
        __syncthreads();
#pragma unroll 1
        for (int i = 1; i + 1 < p.np; ++i) {
          z_mid_pass<T, C, false>(p, i, sc, n, tw);
          __syncthreads();
        }
      }
      z_pair(p.r[p.np - 1], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int tot = n * p.Q * C;
        for (int e = ztid(); e < tot; e += blockDim.x) {
          int b = e >> LC;
          const int row = p.dnb[p.np - 1].div(b), c = e & (C - 1);
          b -= row * p.Q;
          cplx<T>* line = pl + (c0 + row) * C + c;
          cplx<T> f[R], h[R];
          z_last_bfly<T, R, C>(p, line, b, tw, f, st);
          if (X1) {
            z_last_bfly<T, R, C>(p, sc + row * srs + c, b, tw, h);
#pragma unroll
            for (int j = 0; j < R; ++j) f[j] = add(f[j], ik(__ldg(ky + b + p.Q * j), h[j]));
          }
          const int Qp = (p.Q + (p.Q >> p.sh)) * st;
          cplx<T>* q = line + zphys(p, b) * st;
#pragma unroll
          for (int j = 0; j < R; ++j) q[j * Qp] = f[j];
          if constexpr (LOG) {
            const int z = (c0 + row) * C + c;
#pragma unroll
            for (int j = 0; j < R; ++j)
              if (z < nz) log.src[(kx * ny + b + p.Q * j) * nz + z] = f[j];
          }
        }
      });
    }
  }
  // vertical solve, a column per thread; the zero mode on the last warp's first
  // thread, which has no column where the block is larger than the line
  const size_t plane = (size_t)kx * nz * ny;
  double first[kZBatch];
  if (threadIdx.x < ny) z_pivots(first, inv + plane + threadIdx.x, 0, nz, ny);
  __syncthreads();
  double resid = 0.0, compat = 0.0;
  auto source = [&](int k) {
    ZResid<T> r{};
    if constexpr (LOG) {
      const double a = t.kx[kx], b = t.ky[k];
      r = {log.src + (size_t)(kx * ny + k) * nz, t.rho, t.rhoh, arn(mrn(a, a), mrn(b, b)),
           t.dz * t.dz};
    }
    return r;
  };
#pragma unroll 1
  for (int k = threadIdx.x; k < ny; k += blockDim.x) {
    if (kx == 0 && k == 0) continue;
    cplx<T>* col = pl + zphys(p, k) * st;
    const size_t at = plane + k;
    if (k != threadIdx.x) z_pivots(first, inv + at, 0, nz, ny);
    if (sizeof(T) == 4 && lw[(kx * ny + k) >> 5])
      resid += z_sweep<T, true, LOG>(col, nz, ny, inv + at, ad, cd, t.scale, dpd + at, first,
                                     source(k));
    else
      resid += z_sweep<T, false, LOG>(col, nz, ny, inv + at, ad, cd, t.scale, nullptr, first,
                                      source(k));
  }
  if (LOG && kx && 2 * kx != g.nx) resid *= 2.0;  // the half spectrum's other half
  if (kx == 0 && threadIdx.x == ((blockDim.x - 1) & ~31)) {
    resid += z_zero_mode<T, LOG>(pl, nz, t.scale, zw, source(0), t.dz, &compat);
    if constexpr (LOG) log.diag[log.slot_c] = compat;
  }
  if constexpr (LOG) {
    for (int o = 16; o > 0; o >>= 1) resid += __shfl_xor_sync(0xffffffffu, resid, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&log.diag[log.slot_d], resid);
  }
  __syncthreads();

  // inverse lines: i ky' phi^ through the scratch (by groups), phi^ in the plane
#pragma unroll 1
  for (int c0 = out1 ? 0 : nch; c0 < nch + group; c0 += group) {
    const bool both = whole && out1;
    const bool phi = c0 >= nch;  // the plane's turn
    const int n = phi ? nch : min(group, nch - c0);
    cplx<T>* buf = phi ? pl : sc;
    const int bst = phi ? st : C, brs = phi ? C : srs;
    if (c0) __syncthreads();
    z_pair(p.r[p.np - 1], [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int tot = n * p.Q * C;
      const int Qp = (p.Q + (p.Q >> p.sh)) * st;
      for (int e = ztid(); e < tot; e += blockDim.x) {
        int b = e >> LC;
        const int row = p.dnb[p.np - 1].div(b), c = e & (C - 1);
        b -= row * p.Q;
        const cplx<T>* q = pl + ((phi ? 0 : c0) + row) * C + c + zphys(p, b) * st;
        cplx<T> x[R];
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = q[j * Qp];
        if (both) {
          cplx<T> y[R];
#pragma unroll
          for (int j = 0; j < R; ++j) y[j] = x[j];
          z_first_bfly_inv<T, R, C>(p, pl + row * C + c, b, tw, y, st);
        }
        if (!phi) {
#pragma unroll
          for (int j = 0; j < R; ++j) x[j] = ik(__ldg(ky + b + p.Q * j), x[j]);
        }
        z_first_bfly_inv<T, R, C>(p, buf + row * brs + c, b, tw, x, bst);
      }
    });
    __syncthreads();
#pragma unroll 1
    for (int i = p.np - 2; i >= 1; --i) {
      z_mid_pass<T, C, true>(p, i, buf, n, tw, bst, brs);
      if (both) z_mid_pass<T, C, true>(p, i, pl, n, tw, st, C);
      __syncthreads();
    }
    z_last_inv<T, C>(p, buf, n, store(phi ? out0 : out1, phi ? 0 : c0, bst), bst, brs);
    if (both) z_last_inv<T, C>(p, pl, n, store(out0, 0, st), st, C);
    if (phi || both) break;
  }
}

}  // namespace ob
