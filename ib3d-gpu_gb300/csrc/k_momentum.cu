// Momentum predictor: nsMomentum (subNavierStokes.f90:622-1122).
//
// One thread per interior cell of the padded grid; non-fluid cells return at once
// (the reference gathers fluid cells through fluidIndexPtr instead). Per fluid cell:
// staggered transverse-velocity interpolation, third-order upwind convection on
// non-uniform spacing away from walls and immersed-boundary neighbours (else the
// first-order form), second-order diffusion and the explicit pressure gradient,
// then ut = u + dt*(resid + dp/dx) for each component.
//
// Compiled with -fmad=false; each expression keeps the reference's left-to-right
// evaluation so that results are bit-identical to the FP64 oracle.
//
// Bound: the FP64 pipe (1.65 operations per clock and SM). Of about 850 operations a cell
// nearly 500 were divisions, and every divisor depends only on the grid: quotients of two
// grid values come from 1-D tables, rounded as the reference rounds them, and a field value
// is divided by a grid value with div_known, four operations and the same rounding. About
// 470 operations a cell are left: 1.67 -> 0.91 ms at 129x97x75 with the Adams-Bashforth update.
//
// Tables (exact_tables in ib3d_api.cu), t[(axis * kExactTables + tab) * S + m], m the 1-based
// cell index, d the spacings; "own" is the component's axis, "half" a transverse one;
// a divisor takes three tables (b, 1/b in two parts):
//   0 d[m+1]/(d[m]+d[m+1])   1 2/(d[m]+d[m+1])   2 2/(0.5((d[m]+d[m+1])+(d[m]+d[m-1])))
//   divisors: 3 d[m+1]   6 d[m]   9 0.5(d[m]+d[m+1])   12 0.5(d[m]+d[m-1])
//   15 ca6_own d[m+1]   18 2 ck6_own d[m]   21 ca6_half 0.5(d[m]+d[m+1])   24 2 ck6_half 0.5(d[m]+d[m-1])
//   27..33 first-order own: c1, c2, c3, 1/(2 dA), d1, d2, d3;   34..40 the same half
#include "ib3d_internal.cuh"

namespace ib3d {

namespace {

struct Xt {
  const double* t;
  int S;
  __device__ __forceinline__ double operator()(int axis, int tab, int m) const {
    return __ldg(t + (axis * kExactTables + tab) * S + m);
  }
  __device__ __forceinline__ double div(double a, int axis, int tab, int m) const {
    return div_known(a, (*this)(axis, tab, m), (*this)(axis, tab + 1, m), (*this)(axis, tab + 2, m));
  }
};

// Third-order upwind term (subNavierStokes.f90:812-817 and analogues):
// adv*(sum ca*q)/(ca6*dA) + |adv|*(sum ck*q)/(2*ck6*dK). FAM selects the coefficient family at
// compile time so the table pointers stay in the parameter bank (0..2 own axis, 3..5 half).
template <int FAM>
__device__ __forceinline__ double up3(const Grid1D& g, const Xt& T, double adv, int m, double q2, double q1, double q0,
                                      double qm1, double qm2) {
  const double* const* c = g.cc[FAM];
  constexpr int axis = FAM % 3, tab = FAM < 3 ? 15 : 21;
  const double sa = (((c[0][m] * q2 + c[1][m] * q1) + c[2][m] * q0) + c[3][m] * qm1) + c[4][m] * qm2;
  const double sk = (((c[6][m] * q2 + c[7][m] * q1) + c[8][m] * q0) + c[9][m] * qm1) + c[10][m] * qm2;
  return T.div(adv * sa, axis, tab, m) + T.div(fabs(adv) * sk, axis, tab + 3, m);
}

// First-order upwind term (subNavierStokes.f90:847-852 and analogues), al = 1.
template <int AXIS, bool OWN>
__device__ __forceinline__ double up1(const Xt& T, double adv, int m, double qm, double q0, double qp) {
  constexpr int b = OWN ? 27 : 34;
  const double t1 = T.div(adv, AXIS, OWN ? 3 : 9, m) *
                    ((T(AXIS, b, m) * qm - T(AXIS, b + 1, m) * q0) + T(AXIS, b + 2, m) * qp);
  const double t2 = 1.0 * fabs(adv) * T(AXIS, b + 3, m) *
                    ((T(AXIS, b + 4, m) * qm - T(AXIS, b + 5, m) * q0) + T(AXIS, b + 6, m) * qp);
  return t1 - t2;
}

// Second derivative along an axis: lo = q(m-1) - q(m), hi = q(m) - q(m+1).
template <int AXIS, bool OWN>
__device__ __forceinline__ double second(const Xt& T, int m, double lo, double hi) {
  return T(AXIS, OWN ? 1 : 2, m) * (T.div(-hi, AXIS, OWN ? 3 : 9, m) + T.div(lo, AXIS, OWN ? 6 : 12, m));
}

}  // namespace

__global__ void __launch_bounds__(128) k_momentum(Dims d, Grid1D g, const double* __restrict__ tab, int S,
                                                  const double* __restrict__ U, const double* __restrict__ V,
                                                  const double* __restrict__ W, const double* __restrict__ P,
                                                  const unsigned char* __restrict__ C, double* __restrict__ UT,
                                                  double* __restrict__ VT, double* __restrict__ WT, double rev,
                                                  double deltat, double* __restrict__ RU, double* __restrict__ RV,
                                                  double* __restrict__ RW, int ab2) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (unsigned)d.nx * (unsigned)d.ny * (unsigned)d.nz) return;
  const int i = (int)(tid % (unsigned)d.nx) + 2;
  const unsigned t = tid / (unsigned)d.nx;
  const int j = (int)(t % (unsigned)d.ny) + 2, k = (int)(t / (unsigned)d.ny) + 2;
  const long long o = d.at(i, j, k);
  if (C[o] != 0) return;
  const Xt T{tab, S};
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const long long sx = 1, sy = d.NX2, sz = (long long)d.NX2 * d.NY2;
  const double u0 = U[o], v0 = V[o], w0 = W[o];
  const double u22 = U[o - sx] - u0, u4 = u0 - U[o + sx];
  const double u6 = U[o - sy] - u0, u8 = u0 - U[o + sy];
  const double u10 = U[o - sz] - u0, u12 = u0 - U[o + sz];
  const double v4 = V[o - sx] - v0, v6 = v0 - V[o + sx];
  const double v8 = V[o - sy] - v0, v10 = v0 - V[o + sy];
  const double v12 = V[o - sz] - v0, v14 = v0 - V[o + sz];
  const double w6 = W[o - sx] - w0, w8 = w0 - W[o + sx];
  const double w10 = W[o - sy] - w0, w12 = w0 - W[o + sy];
  const double w14 = W[o - sz] - w0, w16 = w0 - W[o + sz];
  const double p0 = P[o];
  const double dpdx = T.div(p0 - P[o + sx], 0, 9, i);   // :779-781
  const double dpdy = T.div(p0 - P[o + sy], 1, 9, j);
  const double dpdz = T.div(p0 - P[o + sz], 2, 9, k);
  const bool noib = C[o + sx] != 2 && C[o - sx] != 2 && C[o + sy] != 2 && C[o - sy] != 2 && C[o + sz] != 2 &&
                    C[o - sz] != 2;
  double cx, cy, cz;

  // ---- u momentum (:792-897)
  {
    const double wx = T(0, 0, i);   // dxr/dx2xr
    const double vu_e = V[o + sx] + wx * (V[o] - V[o + sx]);
    const double vu_w = V[o + sx - sy] + wx * (V[o - sy] - V[o + sx - sy]);
    const double vin = 0.5 * (vu_e + vu_w);
    const double wu_n = W[o + sx] + wx * (W[o] - W[o + sx]);
    const double wu_s = W[o + sx - sz] + wx * (W[o - sz] - W[o + sx - sz]);
    const double win = 0.5 * (wu_n + wu_s);
    if (i != 2 && i < nx && j != 2 && j < ny + 1 && k != 2 && k < nz + 1 && noib) {
      cx = up3<0>(g, T, u0, i, U[o + 2 * sx], U[o + sx], u0, U[o - sx], U[o - 2 * sx]);
      cy = up3<4>(g, T, vin, j, U[o + 2 * sy], U[o + sy], u0, U[o - sy], U[o - 2 * sy]);
      cz = up3<5>(g, T, win, k, U[o + 2 * sz], U[o + sz], u0, U[o - sz], U[o - 2 * sz]);
    } else {
      cx = up1<0, true>(T, u0, i, U[o - sx], u0, U[o + sx]);
      cy = up1<1, false>(T, vin, j, U[o - sy], u0, U[o + sy]);
      cz = up1<2, false>(T, win, k, U[o - sz], u0, U[o + sz]);
    }
    const double d2x = second<0, true>(T, i, u22, u4), d2y = second<1, false>(T, j, u6, u8),
                 d2z = second<2, false>(T, k, u10, u12);
    const double xtt2 = rev * (d2x + d2y + d2z);
    const double resid = -cx - cy - cz + xtt2;
    if (ab2) UT[o] = u0 + deltat * (0.5 * (3.0 * resid - RU[o]) + dpdx);   // nsMomentumAB
    else UT[o] = u0 + deltat * (resid + dpdx);
    if (RU) RU[o] = resid;
  }
  // ---- v momentum (:901-1006)
  {
    const double wy = T(1, 0, j);   // dye/dy2ye
    const double uv_e = U[o + sy] + wy * (U[o] - U[o + sy]);
    const double uv_w = U[o - sx + sy] + wy * (U[o - sx] - U[o - sx + sy]);
    const double uin = 0.5 * (uv_e + uv_w);
    const double wv_n = W[o + sy] + wy * (W[o] - W[o + sy]);
    const double wv_s = W[o + sy - sz] + wy * (W[o - sz] - W[o + sy - sz]);
    const double win = 0.5 * (wv_n + wv_s);
    if (i != 2 && i < nx + 1 && j != 2 && j < ny && k != 2 && k < nz + 1 && noib) {
      cx = up3<3>(g, T, uin, i, V[o + 2 * sx], V[o + sx], v0, V[o - sx], V[o - 2 * sx]);
      cy = up3<1>(g, T, v0, j, V[o + 2 * sy], V[o + sy], v0, V[o - sy], V[o - 2 * sy]);
      cz = up3<5>(g, T, win, k, V[o + 2 * sz], V[o + sz], v0, V[o - sz], V[o - 2 * sz]);
    } else {
      cx = up1<0, false>(T, uin, i, V[o - sx], v0, V[o + sx]);
      cy = up1<1, true>(T, v0, j, V[o - sy], v0, V[o + sy]);
      cz = up1<2, false>(T, win, k, V[o - sz], v0, V[o + sz]);
    }
    const double d2x = second<0, false>(T, i, v4, v6), d2y = second<1, true>(T, j, v8, v10),
                 d2z = second<2, false>(T, k, v12, v14);
    const double ytt2 = rev * (d2x + d2y + d2z);
    const double resid = -cx - cy - cz + ytt2;
    if (ab2) VT[o] = v0 + deltat * (0.5 * (3.0 * resid - RV[o]) + dpdy);   // nsMomentumAB
    else VT[o] = v0 + deltat * (resid + dpdy);
    if (RV) RV[o] = resid;
  }
  // ---- w momentum (:1010-1116)
  {
    const double wz = T(2, 0, k);   // dzt/dz2zt
    const double uw_e = U[o + sz] + wz * (U[o] - U[o + sz]);
    const double uw_w = U[o - sx + sz] + wz * (U[o - sx] - U[o - sx + sz]);
    const double uin = 0.5 * (uw_e + uw_w);
    const double vw_n = V[o + sz] + wz * (V[o] - V[o + sz]);
    const double vw_s = V[o - sy + sz] + wz * (V[o - sy] - V[o - sy + sz]);
    const double vin = 0.5 * (vw_n + vw_s);
    if (i != 2 && i < nx + 1 && j != 2 && j < ny + 1 && k != 2 && k < nz && noib) {
      cx = up3<3>(g, T, uin, i, W[o + 2 * sx], W[o + sx], w0, W[o - sx], W[o - 2 * sx]);
      cy = up3<4>(g, T, vin, j, W[o + 2 * sy], W[o + sy], w0, W[o - sy], W[o - 2 * sy]);
      cz = up3<2>(g, T, w0, k, W[o + 2 * sz], W[o + sz], w0, W[o - sz], W[o - 2 * sz]);
    } else {
      cx = up1<0, false>(T, uin, i, W[o - sx], w0, W[o + sx]);
      cy = up1<1, false>(T, vin, j, W[o - sy], w0, W[o + sy]);
      cz = up1<2, true>(T, w0, k, W[o - sz], w0, W[o + sz]);
    }
    const double d2x = second<0, false>(T, i, w6, w8), d2y = second<1, false>(T, j, w10, w12),
                 d2z = second<2, true>(T, k, w14, w16);
    const double ztt2 = rev * (d2x + d2y + d2z);
    const double resid = -cx - cy - cz + ztt2;
    if (ab2) WT[o] = w0 + deltat * (0.5 * (3.0 * resid - RW[o]) + dpdz);   // nsMomentumAB
    else WT[o] = w0 + deltat * (resid + dpdz);
    if (RW) RW[o] = resid;
  }
}

void launch_momentum(ib3d_ctx* c, bool ab2) {
  PhaseScope ps(c, PH_MOMENTUM);
  c->launches += 1;
  const long long n = (long long)c->d.nx * c->d.ny * c->d.nz;
  const unsigned nb = (unsigned)((n + 127) / 128);
  k_momentum<<<nb, 128, 0, c->st>>>(c->d, c->g, c->d_exact, c->fast_stride, c->u, c->v, c->w, c->p, c->cell, c->ut, c->vt, c->wt,
                                     1.0 / c->prm.re, c->prm.deltat, c->resi[0], c->resi[1], c->resi[2],
                                     ab2 ? 1 : 0);
}

}  // namespace ib3d
