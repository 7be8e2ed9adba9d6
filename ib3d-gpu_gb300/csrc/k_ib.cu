// Immersed-boundary geometry, ghost-point forcing and drag/lift.
//
// Reference: computeSurfaceNorm, tagging, cellCount, computeNormDistance
// (subSearch.f90:80-678), pressureForcing1 / velocityForcing1 (subForcing.f90:2-652),
// stressCal1 / stressCal2 (subStressCal1.f90, subStressCal2.f90).
//
// Compiled with -fmad=false (bit-identical FP64 arithmetic to the serial oracle).
//
// Serial semantics of the forcing. velocityForcing1 reads and writes the same
// arrays: each immersed-boundary (IB) cell writes six ghost faces and its probe
// stencils read faces that earlier cells (or earlier blocks of the same cell) may
// have written, and adjacent IB cells write the same face (the later one wins).
// On a CPU the loop order decides the result; the reference's OpenACC loop races.
// Here every ghost value is an "op" with a serial number (6n + block, or n for the
// pressure). At search time each of an op's eight stencil reads is resolved to
// either the pre-forcing field value or the op that last wrote that face before it
// in serial order (a face of field u has at most two writers: the U(i,j,k) block of
// IB cell (i,j,k) and the U(i-1,j,k) block of IB cell (i+1,j,k)); ops are grouped
// into dependency levels; each level runs as one launch writing to a per-op buffer;
// finally the last writer of each face stores its value. The result equals the
// serial loop's exactly, with no race.
#include <algorithm>

#include "ib3d_internal.cuh"

namespace ib3d {

namespace {

inline unsigned nblk(long long n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }

// l in [lo,hi] with A[l] <= pos < A[l+1], or 0. A is strictly increasing, so this
// is the unique match the reference's linear "keep the last match" scans find.
__device__ __forceinline__ int bracket(const double* A, int lo, int hi, double pos) {
  if (!(pos >= A[lo]) || !(pos < A[hi + 1])) return 0;
  int a = lo, b = hi;
  while (a < b) {
    const int m = (a + b + 1) >> 1;
    if (A[m] <= pos) a = m; else b = m - 1;
  }
  return a;
}

// Trilinear probe value and one-sided quadratic derivative estimates, the common
// block of subForcing.f90:175-215 (and its analogues in subStressCal1.f90).
// f = values at (x0|x1, y0|y1, z0|z1) with x fastest: f[q], q = xbit + 2*ybit + 4*zbit.
// Bound by the warp's count of FP64 instructions (64 cycles each, whatever its lanes do): the
// fifteen divisions by the cell's three widths run through their reciprocals, 4 operations
// each instead of 9, with the same rounded quotients.
__device__ __forceinline__ void probe_eval(const double f[8], const double* X, const double* Y, const double* Z,
                                           int ix, int iy, int iz, double px, double py, double pz,
                                           double out[4]) {
  const double f000 = f[0], f100 = f[1], f010 = f[2], f110 = f[3];
  const double f001 = f[4], f101 = f[5], f011 = f[6], f111 = f[7];
  const double tx = px - X[ix];
  const KnownDiv dX = known(X[ix + 1] - X[ix]);
  const double ty = py - Y[iy];
  const KnownDiv dY = known(Y[iy + 1] - Y[iy]);
  const double tz = pz - Z[iz];
  const KnownDiv dZ = known(Z[iz + 1] - Z[iz]);
  const double x1z1 = f000 + div_known((f100 - f000) * tx, dX);
  const double x2z1 = f010 + div_known((f110 - f010) * tx, dX);
  const double x1z2 = f001 + div_known((f101 - f001) * tx, dX);
  const double x2z2 = f011 + div_known((f111 - f011) * tx, dX);
  const double z1 = x1z1 + div_known((x2z1 - x1z1) * ty, dY);
  const double z2 = x1z2 + div_known((x2z2 - x1z2) * ty, dY);
  const double y1 = x1z1 + div_known((x1z2 - x1z1) * tz, dZ);
  const double y2 = x2z1 + div_known((x2z2 - x2z1) * tz, dZ);
  const double z1x1 = f000 + div_known((f001 - f000) * tz, dZ);
  const double z2x1 = f010 + div_known((f011 - f010) * tz, dZ);
  const double z1x2 = f100 + div_known((f101 - f100) * tz, dZ);
  const double z2x2 = f110 + div_known((f111 - f110) * tz, dZ);
  const double x1 = z1x1 + div_known((z2x1 - z1x1) * ty, dY);
  const double x2 = z1x2 + div_known((z2x2 - z1x2) * ty, dY);
  const double pos = x1 + div_known((x2 - x1) * tx, dX);
  double h2 = fabs(X[ix + 1] - px), h1 = fabs(X[ix] - px);
  out[1] = (h1 * h1 * x2 - h2 * h2 * x1 + (h2 * h2 - h1 * h1) * pos) / (h1 * h2 * (h1 + h2) + 1e-16);
  h2 = fabs(Y[iy + 1] - py); h1 = fabs(Y[iy] - py);
  out[2] = (h1 * h1 * y2 - h2 * h2 * y1 + (h2 * h2 - h1 * h1) * pos) / (h1 * h2 * (h1 + h2) + 1e-16);
  h2 = fabs(Z[iz + 1] - pz); h1 = fabs(Z[iz] - pz);
  out[3] = (h1 * h1 * z2 - h2 * h2 * z1 + (h2 * h2 - h1 * h1) * pos) / (h1 * h2 * (h1 + h2) + 1e-16);
  out[0] = pos;
}

// Velocity ghost-point blocks in subForcing.f90's order (U(i,j,k) :143-224,
// U(i-1,j,k) :227-308, V(i,j,k) :311-393, V(i,j-1,k) :396-478, W(i,j,k) :481-562,
// W(i,j,k-1) :565-646): field, normal-distance slot, node offset, scan extension,
// clamp (+1: idx == n+2 -> n+1 ; -1: idx == 1 -> 2), write-target offset.
struct GhostBlock {
  int field, nd, node[3], scan[3], clamp_axis, clamp_dir, tgt[3];
};
__constant__ GhostBlock c_ghost[6] = {
    {0, 2, {1, 0, 0}, {1, 0, 0}, 0, +1, {0, 0, 0}},
    {0, 1, {0, 0, 0}, {0, 0, 0}, 0, -1, {-1, 0, 0}},
    {1, 4, {0, 1, 0}, {0, 1, 0}, 1, +1, {0, 0, 0}},
    {1, 3, {0, 0, 0}, {0, 0, 0}, 1, -1, {0, -1, 0}},
    {2, 6, {0, 0, 1}, {0, 0, 1}, 2, +1, {0, 0, 0}},
    {2, 5, {0, 0, 0}, {0, 0, 0}, 2, -1, {0, 0, -1}},
};

struct StagCoords {
  const double *X, *Y, *Z;
};
__device__ __forceinline__ StagCoords stag(const Grid1D& g, int field) {
  if (field == 0) return {g.xu, g.yu, g.zu};
  if (field == 1) return {g.xv, g.yv, g.zv};
  if (field == 2) return {g.xw, g.yw, g.zw};
  return {g.xp, g.yp, g.zp};
}

// Geometry of velocity op q = 6n + blk: probe point and pt1, normal distance, nel.
struct OpGeom {
  int i, j, k, nel;
  double sd, pt1, pos[3];
};
__device__ __forceinline__ OpGeom vel_geom(const Grid1D& g, const int* iblist, const int* nelp, const double* nd,
                                           const double* surf, int nib, int nel_tot, int n, int blk) {
  const GhostBlock& gb = c_ghost[blk];
  OpGeom o;
  o.i = iblist[n]; o.j = iblist[nib + n]; o.k = iblist[2 * nib + n];
  o.nel = nelp[n];
  o.sd = nd[gb.nd * nib + n];
  const double diag = sqrt((g.dx[o.i] * g.dx[o.i] + g.dy[o.j] * g.dy[o.j]) + g.dz[o.k] * g.dz[o.k]);
  o.pt1 = 1.5 * diag + (fabs(o.sd) - o.sd) * 0.5;                       // :148
  const StagCoords sc = stag(g, gb.field);
  const int e = o.nel - 1;
  o.pos[0] = sc.X[o.i + gb.node[0]] + o.pt1 * surf[3 * nel_tot + e];    // :151-153
  o.pos[1] = sc.Y[o.j + gb.node[1]] + o.pt1 * surf[4 * nel_tot + e];
  o.pos[2] = sc.Z[o.k + gb.node[2]] + o.pt1 * surf[5 * nel_tot + e];
  return o;
}

}  // namespace

// ------------------------------------------------------------- surface and search

// computeSurfaceNorm (subSearch.f90:95-125).
// flag (may be null) is set where a normal is not finite (a triangle without area).
__global__ void k_surface_norm(const double* __restrict__ nodes, const int* __restrict__ tri, int nn, int ne,
                               double inor, double* __restrict__ surf, int* flag) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int a = tri[e] - 1, b = tri[ne + e] - 1, c = tri[2 * ne + e] - 1;
  const double p1x = nodes[a], p1y = nodes[nn + a], p1z = nodes[2 * nn + a];
  const double p2x = nodes[b], p2y = nodes[nn + b], p2z = nodes[2 * nn + b];
  const double p3x = nodes[c], p3y = nodes[nn + c], p3z = nodes[2 * nn + c];
  surf[e] = ((p2x + p1x) + p3x) / 3.0;
  surf[ne + e] = ((p2y + p1y) + p3y) / 3.0;
  surf[2 * ne + e] = ((p2z + p1z) + p3z) / 3.0;
  const double ca = (p2y - p1y) * (p3z - p1z) - (p3y - p1y) * (p2z - p1z);
  const double cb = (p2z - p1z) * (p3x - p1x) - (p3z - p1z) * (p2x - p1x);
  const double cg = (p2x - p1x) * (p3y - p1y) - (p3x - p1x) * (p2y - p1y);
  surf[6 * ne + e] = ca; surf[7 * ne + e] = cb; surf[8 * ne + e] = cg;
  const double len = sqrt((ca * ca + cb * cb) + cg * cg);
  const double na = (ca / len) * inor, nb = (cb / len) * inor, ng = (cg / len) * inor;
  surf[3 * ne + e] = na;
  surf[4 * ne + e] = nb;
  surf[5 * ne + e] = ng;
  if (flag && !(isfinite(na) && isfinite(nb) && isfinite(ng))) atomicExch(flag, 1);
}

__device__ __forceinline__ double corner_dot(const double* surf, int ne, int e, double x, double y, double z) {
  return ((x - surf[e]) * surf[3 * ne + e] + (y - surf[ne + e]) * surf[4 * ne + e]) +
         (z - surf[2 * ne + e]) * surf[5 * ne + e];
}

// tagging (subSearch.f90:166-249): nearest centroid of each box cell's centre, then
// the signs of the eight corner distances to that element's plane. The reference
// compares dsqrt((dy)^2+(dx)^2+(dz)^2) with strict '<'. Since sqrt is monotone, an
// element whose squared distance is not below the current best's squared distance
// cannot have a strictly smaller rounded root, so the root is only taken for
// candidates that improve the squared distance: the same argmin, bit for bit.
// The result is the lowest index among the elements of smallest rounded distance, whatever
// the order, so elements that cannot attain it need no FP64 arithmetic, which this part
// runs at 1/64 of the FP32 rate (the FP64 scan of every element took 9.6 of 11.3 ms of the
// search at 256x192x192 with 5,120 triangles, an FP32 scan of every element 0.9).
// k_centroid_groups gives the centroids in FP32 relative to the first one, and a sphere
// around each of up to 256 groups of consecutive elements. Per cell: the group with the
// nearest centre is scanned in FP32 for the smallest distance so far, then every group
// whose sphere comes as near as that; elements within the error of the smallest distance
// are queued, and those still within it at the end are evaluated in FP64. Four threads
// share a cell, because the cells near the body's centre, whose distances to all groups
// are alike, would keep single threads busy long after the rest.
// Errors: with L the largest relative coordinate, an FP32 difference is off by at most
// 2^-22 L (two conversions and a subtraction), so a distance by at most 3.5 x 2^-22 L with
// its own rounding, and the nearest element lies within 7 x 2^-22 L of the FP32 minimum;
// the bound used is 16 x 2^-22 L, for the spheres 64 x 2^-22 L, plus 1e-20 for squares that
// underflow. Overflow and NaN pass the filters.
// The cells tagged are the box's (list == nullptr), or the nlist cells of a list inside the
// box (the neighbourhoods of selectiveRetagging); minel is indexed by the cell's position
// in the box either way.
constexpr int kGroups = 256;
// elements per group: at least 32, a multiple of 32, at most kGroups groups
__host__ __device__ __forceinline__ int group_size(int ne) { return ((ne + kGroups - 1) / kGroups + 31) / 32 * 32; }

__device__ __forceinline__ float dist32(const float4 a, float x, float y, float z) {
  const float dx = x - a.x, dy = y - a.y, dz = z - a.z;
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// Relative FP32 centroids c32[0..ne), a sphere per group (centre of the group's bounding
// box, w its radius) behind them, and the largest |coordinate| (bit pattern, reset before).
// One warp per group.
__global__ void k_centroid_groups(const double* __restrict__ surf, int ne, float4* __restrict__ c32,
                                  unsigned* __restrict__ big) {
  const int gs = group_size(ne), lane = threadIdx.x & 31;
  const int gr = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int e0 = gr * gs, e1 = min(ne, e0 + gs);
  if (e0 >= ne) return;
  const double ox = surf[0], oy = surf[ne], oz = surf[2 * ne];
  const float inf = __int_as_float(0x7f800000);
  float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
  for (int e = e0 + lane; e < e1; e += 32) {
    const float v[3] = {(float)(surf[e] - ox), (float)(surf[ne + e] - oy), (float)(surf[2 * ne + e] - oz)};
    c32[e] = make_float4(v[0], v[1], v[2], 0.f);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], v[a]);
      hi[a] = fmaxf(hi[a], v[a]);
    }
  }
  float m = 0.f, c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
    m = fmaxf(m, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
    c[a] = 0.5f * lo[a] + 0.5f * hi[a];
  }
  float r = 0.f;
  for (int e = e0 + lane; e < e1; e += 32) {
    const float d = sqrtf(dist32(c32[e], c[0], c[1], c[2]));
    r = d > r || d != d ? d : r;    // a NaN stays, and keeps the group in
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float x = __shfl_xor_sync(0xffffffffu, r, o);
    r = x > r || x != x ? x : r;
  }
  if (lane == 0) {
    c32[ne + gr] = make_float4(c[0], c[1], c[2], r);
    atomicMax(big, __float_as_uint(m));   // non-negative: the bit patterns order as the numbers
  }
}

__global__ void __launch_bounds__(kBlock) k_tagging(Dims d, Grid1D g, const double* __restrict__ surf, int ne,
                                                    const float4* __restrict__ c32, const unsigned* __restrict__ bigp,
                                                    int bi0, int bj0, int bk0, int bni, int bnj, int bnk,
                                                    const int* __restrict__ list, int nlist,
                                                    unsigned char* __restrict__ cell, int* __restrict__ minel) {
  constexpr int kQueue = 12;
  __shared__ int qe[kQueue][kBlock];     // queued elements, per thread, and their FP32 squared distances
  __shared__ float qd[kQueue][kBlock];
  const int t = threadIdx.x, s = t & 3;  // four threads per cell, thread s its elements s, s + 4, ...
  const unsigned quad = (t & 31) & ~3u;
  const unsigned tid = quad_item(blockIdx.x, blockDim.x, t);
  const unsigned ncell = list ? (unsigned)nlist : (unsigned)bni * (unsigned)bnj * (unsigned)bnk;
  const bool active = tid < ncell;
  const unsigned cid = active ? tid : 0;   // idle threads follow along on cell 0 and store nothing
  int i, j, k;
  if (list) {
    i = list[cid];
    j = list[nlist + cid];
    k = list[2 * nlist + cid];
  } else {
    i = bi0 + (int)(cid % (unsigned)bni);
    const unsigned r = cid / (unsigned)bni;
    j = bj0 + (int)(r % (unsigned)bnj);
    k = bk0 + (int)(r / (unsigned)bnj);
  }
  const double n1x = g.xp[i], n1y = g.yp[j], n1z = g.zp[k];
  const float cx = (float)(n1x - surf[0]), cy = (float)(n1y - surf[ne]), cz = (float)(n1z - surf[2 * ne]);
  const float L = fmaxf(__uint_as_float(*bigp), fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))));
  const float slack = 0x1p-18f * L + 1e-20f, slack_group = 0x1p-16f * L + 1e-20f, up = 1.0f + 0x1p-20f;
  const int gs = group_size(ne), ng = (ne + gs - 1) / gs;
  const float4* sph = c32 + ne;
  const float inf = __int_as_float(0x7f800000);
  float m32 = inf, near2 = inf;          // smallest squared distance so far, and the queue's bound
  double best = 1e14;
  int nel = 0, nq = 0;
  // the queued elements in FP64; together over the warp at the end (one by one each cost the
  // warp a pass of the FP64 pipe)
  auto evaluate = [&]() {
    for (int u = 0; u < nq; ++u) {
      if (qd[u][t] > near2) continue;
      const int e = qe[u][t];
      const double ay = n1y - surf[ne + e], ax = n1x - surf[e], az = n1z - surf[2 * ne + e];
      const double dis = sqrt((ay * ay + ax * ax) + az * az);
      if (dis < best || (dis == best && e + 1 < nel)) { best = dis; nel = e + 1; }
    }
    nq = 0;
  };
  auto scan = [&](int q) {
    const int e1 = min(ne, (q + 1) * gs);
    for (int e0 = q * gs + s; e0 < e1; e0 += 32) {
      float d2[8];
      unsigned cand = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = min(e0 + 4 * u, ne - 1);
        d2[u] = dist32(c32[e], cx, cy, cz);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e0 + 4 * u < e1 && !(d2[u] > near2)) cand |= 1u << u;
      if (cand) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (cand >> u & 1) {
            if (d2[u] < m32) {
              m32 = d2[u];
              const float T = sqrtf(m32) + slack;
              near2 = T * T * up;
            }
            if (nq == kQueue) {            // drop what the bound has left behind
              int n = 0;
              for (int v = 0; v < kQueue; ++v)
                if (!(qd[v][t] > near2)) {
                  qe[n][t] = qe[v][t];
                  qd[n][t] = qd[v][t];
                  ++n;
                }
              nq = n;
              if (nq == kQueue) evaluate();
            }
            qe[nq][t] = e0 + 4 * u;
            qd[nq][t] = d2[u];
            ++nq;
          }
      }
    }
    // the four threads share the smallest distance
    m32 = fminf(m32, __shfl_xor_sync(0xfu << quad, m32, 1));
    m32 = fminf(m32, __shfl_xor_sync(0xfu << quad, m32, 2));
    const float T = sqrtf(m32) + slack;
    near2 = T * T * up;
  };
  float c2 = inf;
  int g0 = 0;
#pragma unroll 4
  for (int q = s; q < ng; q += 4) {
    const float d2 = dist32(sph[q], cx, cy, cz);
    if (d2 < c2) { c2 = d2; g0 = q; }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    const float x = __shfl_xor_sync(0xffffffffu, c2, o);
    const int y = __shfl_xor_sync(0xffffffffu, g0, o);
    if (x < c2 || (x == c2 && y < g0)) { c2 = x; g0 = y; }
  }
  scan(g0);
  for (int q0 = 0; q0 < ng; q0 += 4) {
    const int q = q0 + s;
    bool in = false;
    if (q < ng && q != g0) {
      const float4 sp = sph[q];
      const float tr = sqrtf(m32) + slack_group + sp.w;
      in = !(dist32(sp, cx, cy, cz) > tr * tr * up);
    }
    const unsigned m = __ballot_sync(0xffffffffu, in) >> quad;
#pragma unroll 1
    for (int u = 0; u < 4; ++u)
      if (m >> u & 1) scan(q0 + u);
  }
  evaluate();
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    const double x = __shfl_xor_sync(0xffffffffu, best, o);
    const int y = __shfl_xor_sync(0xffffffffu, nel, o);
    if (y != 0 && (nel == 0 || x < best || (x == best && y < nel))) { best = x; nel = y; }
  }
  if (nel == 0) nel = 1;   // no element within 1e14
  // the signs of the eight corners' distances to the element's plane, two per thread
  const double x = s & 1 ? g.x1[i + 1] : g.x1[i], z = s & 2 ? g.z1[k + 1] : g.z1[k];
  const double d0 = corner_dot(surf, ne, nel - 1, x, g.y1[j], z), d1 = corner_dot(surf, ne, nel - 1, x, g.y1[j + 1], z);
  const double thr = -1e-16;
  const bool all_in = (__ballot_sync(0xffffffffu, d0 <= thr && d1 <= thr) >> quad & 15u) == 15u;
  const bool all_out = (__ballot_sync(0xffffffffu, d0 > thr && d1 > thr) >> quad & 15u) == 15u;
  if (active && s == 0) {
    cell[d.at(i, j, k)] = all_in ? 1 : (all_out ? 0 : 2);
    minel[(i - bi0) + bni * ((j - bj0) + bnj * (k - bk0))] = nel;
  }
}

// Bounding box of the IB list: {min i, max i, min j, max j, min k, max k}, out[] set
// to {INT_MAX, INT_MIN, ...} before the launch.
__global__ void k_ib_bounds(const int* __restrict__ iblist, int nib, int* __restrict__ out) {
  int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-0x7fffffff, -0x7fffffff, -0x7fffffff};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nib; n += gridDim.x * blockDim.x)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int v = iblist[a * nib + n];
      lo[a] = min(lo[a], v);
      hi[a] = max(hi[a], v);
    }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = min(lo[a], __shfl_down_sync(0xffffffffu, lo[a], o));
      hi[a] = max(hi[a], __shfl_down_sync(0xffffffffu, hi[a], o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&out[2 * a], lo[a]);
      atomicMax(&out[2 * a + 1], hi[a]);
    }
  }
}

// selectiveRetagging's neighbourhoods (subSearch.f90:355-358): cells i1-2..i1+3,
// j1-2..j1+3, k1-2..k1+3 of every IB cell (i1,j1,k1), clipped to the box (the
// neighbourhoods' bounding box clipped to the interior), marked in a box-shaped mask.
// Overlapping neighbourhoods write the same value.
__global__ void k_mark_neighbourhoods(const int* __restrict__ iblist, int nib, int bi0, int bj0, int bk0, int bni,
                                      int bnj, int bnk, unsigned char* __restrict__ mask) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (unsigned)nib * 216u) return;
  const int n = (int)(tid / 216u), o = (int)(tid % 216u);
  const int i = iblist[n] - 2 + o % 6, j = iblist[nib + n] - 2 + (o / 6) % 6, k = iblist[2 * nib + n] - 2 + o / 36;
  const int li = i - bi0, lj = j - bj0, lk = k - bk0;
  if (li >= 0 && li < bni && lj >= 0 && lj < bnj && lk >= 0 && lk < bnk) mask[li + bni * (lj + bnj * lk)] = 1;
}

// Compaction of the marked cells of a box-shaped mask into a list (i block, j block,
// k block); same three passes as the IB compaction below.
__global__ void k_mask_blockcount(const unsigned char* __restrict__ mask, unsigned nbox, long long* bcount) {
  __shared__ int s;
  if (threadIdx.x == 0) s = 0;
  __syncthreads();
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool f = t < nbox && mask[t];
  const unsigned bal = __ballot_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && bal) atomicAdd(&s, __popc(bal));
  __syncthreads();
  if (threadIdx.x == 0) bcount[blockIdx.x] = s;
}
__global__ void k_mask_scatter(const unsigned char* __restrict__ mask, unsigned nbox, int bi0, int bj0, int bk0,
                               int bni, int bnj, const long long* __restrict__ boff, int nlist,
                               int* __restrict__ list) {
  __shared__ int wsum[kBlock / 32];
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool f = t < nbox && mask[t];
  const unsigned bal = __ballot_sync(0xffffffffu, f);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) wsum[wid] = __popc(bal);
  __syncthreads();
  int before = 0;
  for (int q = 0; q < wid; ++q) before += wsum[q];
  before += __popc(bal & ((1u << lane) - 1u));
  if (f) {
    const long long n = boff[blockIdx.x] + before;
    if (n < nlist) {
      list[n] = bi0 + (int)(t % (unsigned)bni);
      const unsigned r = t / (unsigned)bni;
      list[nlist + n] = bj0 + (int)(r % (unsigned)bnj);
      list[2 * nlist + n] = bk0 + (int)(r / (unsigned)bnj);
    }
  }
}

// Cell counts over the interior (subSearch.f90:259-270) and the red/black split of
// the fluid cells (subSearch.f90:557-567): {fluid, solid, ib, red, black}.
__global__ void __launch_bounds__(kBlock) k_count(Dims d, const unsigned char* __restrict__ cell,
                                                  unsigned long long* counts) {
  __shared__ unsigned int sc[5];
  if (threadIdx.x < 5) sc[threadIdx.x] = 0;
  __syncthreads();
  unsigned n[5] = {0, 0, 0, 0, 0};
  const unsigned total = (unsigned)d.nx * (unsigned)d.ny * (unsigned)d.nz;
  for (unsigned tid = blockIdx.x * blockDim.x + threadIdx.x; tid < total; tid += gridDim.x * blockDim.x) {
    const int i = (int)(tid % (unsigned)d.nx) + 2;
    const unsigned t = tid / (unsigned)d.nx;
    const int j = (int)(t % (unsigned)d.ny) + 2, k = (int)(t / (unsigned)d.ny) + 2;
    const unsigned char c = cell[d.at(i, j, k)];
    n[0] += c == 0;
    n[1] += c == 1;
    n[2] += c == 2;
    n[3] += c == 0 && ((i + j + k) & 1);
    n[4] += c == 0 && !((i + j + k) & 1);
  }
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const unsigned s = __reduce_add_sync(0xffffffffu, n[q]);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(&sc[q], s);
  }
  __syncthreads();
  if (threadIdx.x < 5 && sc[threadIdx.x]) atomicAdd(&counts[threadIdx.x], (unsigned long long)sc[threadIdx.x]);
}

// Lexicographic compaction of the IB cells (cellCount, subSearch.f90:532-553): the
// box is scanned with i fastest, then j, then k, which is the reference's loop
// order. Pass 1 counts per block, pass 2 scans the block counts, pass 3 writes.
__device__ __forceinline__ bool box_is_ib(const Dims& d, const unsigned char* cell, unsigned tid, int bi0, int bj0,
                                          int bk0, int bni, int bnj, unsigned nbox, int& i, int& j, int& k) {
  if (tid >= nbox) return false;
  i = bi0 + (int)(tid % (unsigned)bni);
  const unsigned t = tid / (unsigned)bni;
  j = bj0 + (int)(t % (unsigned)bnj);
  k = bk0 + (int)(t / (unsigned)bnj);
  if (i < 2 || i > d.nx + 1 || j < 2 || j > d.ny + 1 || k < 2 || k > d.nz + 1) return false;
  return cell[d.at(i, j, k)] == 2;
}
__global__ void k_ib_blockcount(Dims d, const unsigned char* __restrict__ cell, int bi0, int bj0, int bk0, int bni,
                                int bnj, unsigned nbox, long long* bcount) {
  __shared__ int s;
  if (threadIdx.x == 0) s = 0;
  __syncthreads();
  int i, j, k;
  const bool f = box_is_ib(d, cell, blockIdx.x * blockDim.x + threadIdx.x, bi0, bj0, bk0, bni, bnj, nbox, i, j, k);
  const unsigned bal = __ballot_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && bal) atomicAdd(&s, __popc(bal));
  __syncthreads();
  if (threadIdx.x == 0) bcount[blockIdx.x] = s;
}
__global__ void k_exclusive_scan(long long* a, int n, long long* total) {
  // single block; a sequential carry over 1024-wide chunks
  __shared__ long long buf[1024];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int q = base + threadIdx.x;
    const long long x = q < n ? a[q] : 0;
    buf[threadIdx.x] = x;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
      const long long y = threadIdx.x >= off ? buf[threadIdx.x - off] : 0;
      __syncthreads();
      buf[threadIdx.x] += y;
      __syncthreads();
    }
    if (q < n) a[q] = carry + buf[threadIdx.x] - x;
    __syncthreads();
    if (threadIdx.x == 1023) carry += buf[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}
__global__ void k_ib_scatter(Dims d, const unsigned char* __restrict__ cell, int bi0, int bj0, int bk0, int bni,
                             int bnj, unsigned nbox, const long long* __restrict__ boff, int nib,
                             int* __restrict__ iblist) {
  __shared__ int wsum[kBlock / 32];
  int i = 0, j = 0, k = 0;
  const bool f = box_is_ib(d, cell, blockIdx.x * blockDim.x + threadIdx.x, bi0, bj0, bk0, bni, bnj, nbox, i, j, k);
  const unsigned bal = __ballot_sync(0xffffffffu, f);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) wsum[wid] = __popc(bal);
  __syncthreads();
  int before = 0;
  for (int q = 0; q < wid; ++q) before += wsum[q];
  before += __popc(bal & ((1u << lane) - 1u));
  if (f) {
    const long long n = boff[blockIdx.x] + before;
    if (n < nib) { iblist[n] = i; iblist[nib + n] = j; iblist[2 * nib + n] = k; }
  }
}

// computeNormDistance (subSearch.f90:621-672) plus the IB index map.
__global__ void k_normdist(Dims d, Grid1D g, const double* __restrict__ surf, int ne, const int* __restrict__ iblist,
                           int nib, const int* __restrict__ minel, int bi0, int bj0, int bk0, int bni, int bnj,
                           int* __restrict__ nelp, double* __restrict__ nd, int* __restrict__ ibmap) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nib) return;
  const int i = iblist[n], j = iblist[nib + n], k = iblist[2 * nib + n];
  const double n1x = g.xp[i], n2x = g.x1[i], n3x = g.x1[i + 1];
  const double n1y = g.yp[j], n2y = g.y1[j], n3y = g.y1[j + 1];
  const double n1z = g.zp[k], n2z = g.z1[k], n3z = g.z1[k + 1];
  const int m = minel[(i - bi0) + bni * ((j - bj0) + bnj * (k - bk0))];
  nelp[n] = m;
  const int e = m - 1;
  nd[0 * nib + n] = corner_dot(surf, ne, e, n1x, n1y, n1z);
  nd[1 * nib + n] = corner_dot(surf, ne, e, n2x, n1y, n1z);
  nd[2 * nib + n] = corner_dot(surf, ne, e, n3x, n1y, n1z);
  nd[3 * nib + n] = corner_dot(surf, ne, e, n1x, n2y, n1z);
  nd[4 * nib + n] = corner_dot(surf, ne, e, n1x, n3y, n1z);
  nd[5 * nib + n] = corner_dot(surf, ne, e, n1x, n1y, n2z);
  nd[6 * nib + n] = corner_dot(surf, ne, e, n1x, n1y, n3z);
  ibmap[d.at(i, j, k)] = n;
}

// --------------------------------------------------------------- forcing schedule

// Serial number of the op that writes face (a,b,c) of `field` through IB cell
// (ci,cj,ck) with block blk, or -1 when that cell is not an IB cell.
__device__ __forceinline__ long long writer(const Dims& d, const int* ibmap, int ci, int cj, int ck, int blk) {
  if (ci < 2 || ci > d.nx + 1 || cj < 2 || cj > d.ny + 1 || ck < 2 || ck > d.nz + 1) return -1;
  const int n = ibmap[d.at(ci, cj, ck)];
  return n < 0 ? -1 : 6ll * n + blk;
}
// The two possible writers of face (a,b,c) of a velocity field: the "own" block of
// IB cell (a,b,c) and the "minus" block of the next IB cell along the field's axis.
__device__ __forceinline__ void face_writers(const Dims& d, const int* ibmap, int field, int a, int b, int c,
                                             long long w[2]) {
  w[0] = writer(d, ibmap, a, b, c, 2 * field);
  w[1] = writer(d, ibmap, a + (field == 0), b + (field == 1), c + (field == 2), 2 * field + 1);
}

// Builds the velocity ops: brackets, clamps, the eight read indices with their
// sources, the target and whether the op is its target's last writer.
__global__ void k_sched_vel(Dims d, Grid1D g, const int* __restrict__ iblist, const int* __restrict__ nelp,
                            const double* __restrict__ nd, const double* __restrict__ surf, int nib, int ne,
                            const int* __restrict__ ibmap, int* __restrict__ brk, int* __restrict__ rd_idx,
                            int* __restrict__ rd_src, int* __restrict__ tgt, unsigned char* __restrict__ fin,
                            int* err, int* deps) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= 6ll * nib) return;
  const int n = (int)(q / 6), blk = (int)(q % 6);
  const GhostBlock& gb = c_ghost[blk];
  const OpGeom o = vel_geom(g, iblist, nelp, nd, surf, nib, ne, n, blk);
  const StagCoords sc = stag(g, gb.field);
  const int nn[3] = {d.nx, d.ny, d.nz};
  const double* A[3] = {sc.X, sc.Y, sc.Z};
  int br[3];
  for (int a = 0; a < 3; ++a) {
    br[a] = bracket(A[a], 1, nn[a] + 1 + gb.scan[a], o.pos[a]);
    if (br[a] == 0) { atomicExch(err, 1); br[a] = 2; }
  }
  const int ca = gb.clamp_axis;
  if (gb.clamp_dir > 0) { if (br[ca] == nn[ca] + 2) br[ca] = nn[ca] + 1; }    // e.g. :171
  else { if (br[ca] == 1) br[ca] = 2; }                                       // e.g. :252
  // A bracket in the first ghost layer would address field index 0 (the reference
  // would read outside its array): report the probe as off the grid and use a safe cell.
  if (br[gb.field] < 2) { atomicExch(err, 1); br[gb.field] = 2; }
  brk[3 * q] = br[0]; brk[3 * q + 1] = br[1]; brk[3 * q + 2] = br[2];
  const int a0 = br[0] - (gb.field == 0), b0 = br[1] - (gb.field == 1), c0 = br[2] - (gb.field == 2);
  for (int r = 0; r < 8; ++r) {
    const int a = a0 + (r & 1), b = b0 + ((r >> 1) & 1), c = c0 + (r >> 2);
    rd_idx[8 * q + r] = (int)d.at(a, b, c);
    long long w[2];
    face_writers(d, ibmap, gb.field, a, b, c, w);
    long long src = -1;
    for (int s = 0; s < 2; ++s)
      if (w[s] >= 0 && w[s] < q && w[s] > src) src = w[s];
    rd_src[8 * q + r] = (int)src;
    if (src >= 0) *deps = 1;
  }
  const int ta = o.i + gb.tgt[0], tb = o.j + gb.tgt[1], tc = o.k + gb.tgt[2];
  tgt[q] = (int)d.at(ta, tb, tc);
  long long w[2];
  face_writers(d, ibmap, gb.field, ta, tb, tc, w);
  fin[q] = (w[0] > q || w[1] > q) ? 0 : 1;
}

// Pressure ops: one per IB cell (subForcing.f90:18-98); p(a,b,c) has one writer,
// the IB cell (a,b,c) itself.
__global__ void k_sched_p(Dims d, Grid1D g, const int* __restrict__ iblist, const int* __restrict__ nelp,
                          const double* __restrict__ nd, const double* __restrict__ surf, int nib, int ne,
                          const int* __restrict__ ibmap, int* __restrict__ brk, int* __restrict__ rd_idx,
                          int* __restrict__ rd_src, int* __restrict__ tgt, unsigned char* __restrict__ fin,
                          int* err, int* deps) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nib) return;
  const int i = iblist[n], j = iblist[nib + n], k = iblist[2 * nib + n];
  const int e = nelp[n] - 1;
  const double sd = nd[n];
  const double pt1 = 1.5 * sqrt((g.dx[i] * g.dx[i] + g.dy[j] * g.dy[j]) + g.dz[k] * g.dz[k]) + (fabs(sd) - sd) * 0.5;
  const double pos[3] = {g.xp[i] + pt1 * surf[3 * ne + e], g.yp[j] + pt1 * surf[4 * ne + e],
                         g.zp[k] + pt1 * surf[5 * ne + e]};
  const double* A[3] = {g.xp, g.yp, g.zp};
  const int nn[3] = {d.nx, d.ny, d.nz};
  int br[3];
  for (int a = 0; a < 3; ++a) {
    br[a] = bracket(A[a], 1, nn[a] + 1, pos[a]);
    if (br[a] == 0) { atomicExch(err, 1); br[a] = 2; }
  }
  brk[3 * n] = br[0]; brk[3 * n + 1] = br[1]; brk[3 * n + 2] = br[2];
  for (int r = 0; r < 8; ++r) {
    const int a = br[0] + (r & 1), b = br[1] + ((r >> 1) & 1), c = br[2] + (r >> 2);
    const long long L = d.at(a, b, c);
    rd_idx[8 * n + r] = (int)L;
    int src = -1;
    if (a >= 2 && a <= d.nx + 1 && b >= 2 && b <= d.ny + 1 && c >= 2 && c <= d.nz + 1) {
      const int m = ibmap[L];
      if (m >= 0 && m < n) src = m;
    }
    rd_src[8 * n + r] = src;
    if (src >= 0) *deps = 1;
  }
  tgt[n] = (int)d.at(i, j, k);
  fin[n] = 1;
}

// ------------------------------------------------------------ forcing execution

// One dependency level of velocityForcing1 (subForcing.f90:143-646 per op).
__global__ void k_force_vel(Grid1D g, const int* __restrict__ order, int off, int cnt,
                            const int* __restrict__ iblist, const int* __restrict__ nelp,
                            const double* __restrict__ nd, const double* __restrict__ surf, int nib, int ne,
                            const int* __restrict__ brk, const int* __restrict__ rd_idx,
                            const int* __restrict__ rd_src, const double* __restrict__ ut,
                            const double* __restrict__ vt, const double* __restrict__ wt, Motion mo,
                            double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const int q = order ? order[off + t] : t;   // null: one level holds every op
  const int n = q / 6, blk = q % 6;
  const GhostBlock& gb = c_ghost[blk];
  const OpGeom o = vel_geom(g, iblist, nelp, nd, surf, nib, ne, n, blk);
  const StagCoords sc = stag(g, gb.field);
  const double* F = gb.field == 0 ? ut : gb.field == 1 ? vt : wt;
  double f[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int s = rd_src[8 * q + r];
    f[r] = s >= 0 ? out[s] : F[rd_idx[8 * q + r]];
  }
  double pe[4];
  probe_eval(f, sc.X, sc.Y, sc.Z, brk[3 * q], brk[3 * q + 1], brk[3 * q + 2], o.pos[0], o.pos[1], o.pos[2], pe);
  const int e = o.nel - 1;
  const double dndn = pe[1] * surf[3 * ne + e] + pe[2] * surf[4 * ne + e] + pe[3] * surf[5 * ne + e];
  const double n1 = o.pt1 + o.sd;
  const double surfv = mo.moving ? mo.vel[gb.field] : 0.0;           // usurf = u_curr (:144) or 0 (:145)
  const double cval = surfv;
  const double bval = 2.0 / n1 * (pe[0] - surfv) - dndn;              // :222
  const double aval = dndn / n1 - (pe[0] - surfv) / (n1 * n1);        // :223
  out[q] = aval * (o.sd * o.sd) + bval * o.sd + cval;                 // :224
}

// One dependency level of pressureForcing1 (subForcing.f90:18-98); dpdn = 0 for a
// fixed body (:11), the body acceleration along the normal for a moving one (:20).
__global__ void k_force_p(Grid1D g, const int* __restrict__ order, int off, int cnt, const int* __restrict__ iblist,
                          const int* __restrict__ nelp, const double* __restrict__ nd,
                          const double* __restrict__ surf, int nib, int ne, const int* __restrict__ brk,
                          const int* __restrict__ rd_idx, const int* __restrict__ rd_src,
                          const double* __restrict__ p, Motion mo, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const int n = order ? order[off + t] : t;
  const int i = iblist[n], j = iblist[nib + n], k = iblist[2 * nib + n];
  const int e = nelp[n] - 1;
  const double sd = nd[n];
  const double pt1 = 1.5 * sqrt((g.dx[i] * g.dx[i] + g.dy[j] * g.dy[j]) + g.dz[k] * g.dz[k]) + (fabs(sd) - sd) * 0.5;
  const double px = g.xp[i] + pt1 * surf[3 * ne + e];
  const double py = g.yp[j] + pt1 * surf[4 * ne + e];
  const double pz = g.zp[k] + pt1 * surf[5 * ne + e];
  double f[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int s = rd_src[8 * n + r];
    f[r] = s >= 0 ? out[s] : p[rd_idx[8 * n + r]];
  }
  double pe[4];
  probe_eval(f, g.xp, g.yp, g.zp, brk[3 * n], brk[3 * n + 1], brk[3 * n + 2], px, py, pz, pe);
  const double dpdn = mo.moving ? (mo.acc[0] * surf[3 * ne + e] + mo.acc[1] * surf[4 * ne + e]) +
                                      mo.acc[2] * surf[5 * ne + e]
                                : 0.0;
  const double dpdn_e = pe[1] * surf[3 * ne + e] + pe[2] * surf[4 * ne + e] + pe[3] * surf[5 * ne + e];
  const double n1 = pt1 + sd;
  const double bval = dpdn;
  const double aval = (dpdn_e - dpdn) / (2.0 * n1);                  // :95
  const double cval = pe[0] - (dpdn_e + dpdn) * n1 * 0.5;            // :96
  out[n] = aval * (sd * sd) + bval * sd + cval;                      // :98
}

// Stores each face's last-writer value (after every level has run).
__global__ void k_force_scatter(const unsigned char* __restrict__ fin, int nops, const int* __restrict__ tgt,
                                const double* __restrict__ out, int vel, double* f0, double* f1, double* f2) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nops || !fin[q]) return;
  double* F = f0;
  if (vel) {
    const int field = (q % 6) >> 1;
    F = field == 0 ? f0 : field == 1 ? f1 : f2;
  }
  F[tgt[q]] = out[q];
}

// ------------------------------------------------------------------- drag / lift

// Per-element terms of stressCal1/2 (subStressCal1.f90:85-434): viscous traction and
// pressure force from the probe at one cell diagonal along the normal. Probe cells
// are found on the first call and cached (stressCal2 reuses them, :81-83 etc.).
// Four threads per element, one per probed field: each probe is a chain of some 20 FP64
// divisions, and 5,120 elements of one thread each filled 20 of the SMs (with the sum below
// 0.35 ms; now 0.1).
__global__ void __launch_bounds__(64) k_stress_elem(Dims d, Grid1D g, const double* __restrict__ surf, int ne, int first,
                                                    int* __restrict__ scache, const double* __restrict__ ut,
                                                    const double* __restrict__ vt, const double* __restrict__ wt,
                                                    const double* __restrict__ p, double inv_re,
                                                    double* __restrict__ contrib, int* err) {
  const int e0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, c = threadIdx.x & 3;
  const bool active = e0 < ne;
  const int e = active ? e0 : ne - 1;   // idle threads follow along on the last element and store nothing
  const int lead = (threadIdx.x & 31) & ~3;
  const int nn[3] = {d.nx, d.ny, d.nz};
  const double xs = surf[e], ys = surf[ne + e], zs = surf[2 * ne + e];
  const double ca = surf[3 * ne + e], cb = surf[4 * ne + e], cg = surf[5 * ne + e];
  int cell = 0;   // thread c < 3: the element's cell along axis c
  if (c < 3) {
    if (first) {
      cell = bracket(c == 0 ? g.x1 : c == 1 ? g.y1 : g.z1, 2, c == 0 ? d.nx + 1 : c == 1 ? d.ny + 1 : d.nz + 1,
                     c == 0 ? xs : c == 1 ? ys : zs);                  // :89-105
      if (!cell) { if (active) atomicExch(err, 1); cell = 2; }
      if (active) scache[15 * e + c] = cell;
    } else {
      cell = scache[15 * e + c];
    }
  }
  const int ic = __shfl_sync(0xffffffffu, cell, lead), jc = __shfl_sync(0xffffffffu, cell, lead + 1),
            kc = __shfl_sync(0xffffffffu, cell, lead + 2);
  const double dX = g.x1[ic + 1] - g.x1[ic], dY = g.y1[jc + 1] - g.y1[jc], dZ = g.z1[kc + 1] - g.z1[kc];
  const double diagdis = sqrt((dX * dX + dY * dY) + dZ * dZ);           // :119
  const double px = xs + diagdis * ca, py = ys + diagdis * cb, pz = zs + diagdis * cg;
  const StagCoords sc = stag(g, c);
  int br[3];
  if (first) {
    const double ppos[3] = {px, py, pz};
    const double* A[3] = {sc.X, sc.Y, sc.Z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      br[a] = bracket(A[a], 2, nn[a] + 1, ppos[a]);                     // e.g. :135-145
      if (!br[a]) { if (active) atomicExch(err, 1); br[a] = 2; }
      if (active) scache[15 * e + 3 + 3 * c + a] = br[a];
    }
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) br[a] = scache[15 * e + 3 + 3 * c + a];
  }
  const double* F = c == 0 ? ut : c == 1 ? vt : c == 2 ? wt : p;
  const int a0 = br[0] - (c == 0), b0 = br[1] - (c == 1), c0 = br[2] - (c == 2);
  double f[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) f[r] = F[d.at(a0 + (r & 1), b0 + ((r >> 1) & 1), c0 + (r >> 2))];
  double pe[4];
  probe_eval(f, sc.X, sc.Y, sc.Z, br[0], br[1], br[2], px, py, pz, pe);
  const double dn_e = pe[1] * ca + pe[2] * cb + pe[3] * cg;
  const double dn = (2.0 / diagdis) * (pe[0] - 0.0) - dn_e;             // :195, :260, :324 (threads 0..2)
  const double dnds[3] = {__shfl_sync(0xffffffffu, dn, lead), __shfl_sync(0xffffffffu, dn, lead + 1),
                          __shfl_sync(0xffffffffu, dn, lead + 2)};
  if (active && c == 3) {
    const double a3 = surf[6 * ne + e], b3 = surf[7 * ne + e], g3 = surf[8 * ne + e];
    const double alen = sqrt((a3 * a3 + b3 * b3) + g3 * g3);           // :327-331
    const double area = alen / 2.0;
    const double dot = dnds[0] * ca + dnds[1] * cb + dnds[2] * cg;
    const double stx1 = dnds[0] - dot * ca;                           // :335-337
    const double sty1 = dnds[1] - dot * cb;
    const double dpdn = 0.0;
    const double cval = pe[0] - (dn_e + dpdn) * diagdis * 0.5;        // :415
    const double f_surf = cval * area;
    contrib[0 * ne + e] = inv_re * stx1 * area;                       // shear_x_force :341
    contrib[1 * ne + e] = -f_surf * ca;                               // f_surf_x :421
    contrib[2 * ne + e] = inv_re * sty1 * area;                       // shear_y_force :343
    contrib[3 * ne + e] = -f_surf * cb;                               // f_surf_y :423
    contrib[4 * ne + e] = area;
    contrib[5 * ne + e] = 0.5 * fabs(b3);                             // area_xz :330
    contrib[6 * ne + e] = 0.5 * fabs(a3);                             // area_yz :329
  }
}

__device__ __forceinline__ void stress_coefficients(const double* s, double* coef) {
  const double area_Sx = 0.5 * s[5], area_Sy = 0.5 * s[6];
  coef[0] = 2.0 * (s[0] / area_Sx);
  coef[1] = 2.0 * (s[1] / area_Sy);
  coef[2] = 2.0 * (s[2] / area_Sy);
  coef[3] = 2.0 * (s[3] / area_Sx);
}

// Element-order sums (the serial order of the reference's loop, so the sums are
// bit-identical to the oracle) and the coefficients (subStressCal1.f90:428-450). A sum is
// one chain of FP64 additions, about 85 cycles each on this part: 0.21 ms for 5,120
// elements; the block brings the terms into shared memory ahead of the seven adding threads.
constexpr int kSumTile = 256, kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_stress_sum(const double* __restrict__ contrib, int ne, double* coef) {
  __shared__ double tile[2][7][kSumTile + 1];   // the seven rows in different banks
  __shared__ double s[7];
  const int t = threadIdx.x;
  auto fetch = [&](int base, double (&v)[7]) {
#pragma unroll
    for (int q = 0; q < 7; ++q) v[q] = base + t < ne ? contrib[(long long)q * ne + base + t] : 0.0;
  };
  double v[7], acc = 0.0;
  fetch(0, v);
  int buf = 0;
  for (int base = 0; base < ne; base += kSumTile, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < 7; ++q) tile[buf][q][t] = v[q];
    __syncthreads();
    if (base + kSumTile < ne) fetch(base + kSumTile, v);
    if (t < 7) {
      const double* c = tile[buf][t];
      const int cnt = min(kSumTile, ne - base);
#pragma unroll 16
      for (int e = 0; e < cnt; ++e) acc = acc + c[e];
    }
  }
  if (t < 7) s[t] = acc;
  __syncthreads();
  if (t == 0) stress_coefficients(s, coef);
}

// The same sums in a fixed tree order, for the forms whose results may differ from the
// reference's arithmetic by rounding (IB3D_PREC_FP32DC, IB3D_PREC_FP64_FAST). A block per sum
// (one block for all seven was bound by its SM's FP64 pipe: 14 us for 5,120 elements); the
// last to finish works out the coefficients. sums: coef[8 .. 14]; coef[15] counts the blocks
// and is left at 0.
constexpr int kTreeThreads = 512;
__global__ void __launch_bounds__(kTreeThreads) k_stress_sum_tree(const double* __restrict__ contrib, int ne, double* coef) {
  __shared__ double w[kTreeThreads / 32];
  const int t = threadIdx.x, q = blockIdx.x;
  double a = 0.0;
  for (int e = t; e < ne; e += kTreeThreads) a += contrib[(long long)q * ne + e];
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if ((t & 31) == 0) w[t >> 5] = a;
  __syncthreads();
  if (t < 32) {
    double x = t < kTreeThreads / 32 ? w[t] : 0.0;
    for (int o = kTreeThreads / 64; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (t == 0) {
      int* done = reinterpret_cast<int*>(coef + 15);
      coef[8 + q] = x;
      __threadfence();
      if (atomicAdd(done, 1) == 6) {
        __threadfence();
        double s[7];
#pragma unroll
        for (int r = 0; r < 7; ++r) s[r] = __ldcg(coef + 8 + r);
        stress_coefficients(s, coef);
        *done = 0;
      }
    }
  }
}

// ------------------------------------------------------------------- host side

// shiftSurfaceNodesMovingbody's node loop (subSearch.f90:64-73): x = xr + xmove.
__global__ void k_shift_nodes(double* __restrict__ nodes, int nn, double dx, double dy, double dz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const double xr = nodes[i], yr = nodes[nn + i], zr = nodes[2 * nn + i];
  nodes[i] = xr + dx;
  nodes[nn + i] = yr + dy;
  nodes[2 * nn + i] = zr + dz;
}

int run_move_body(ib3d_ctx* c, double dx, double dy, double dz) {
  k_shift_nodes<<<nblk(c->nnodes), kBlock, 0, c->st>>>(c->d_nodes, (int)c->nnodes, dx, dy, dz);
  IB3D_CUDA(c, cudaGetLastError());
  c->launches += 2;
  return run_surface_norm(c, nullptr);
}

int run_surface_norm(ib3d_ctx* c, int* flag) {
  k_surface_norm<<<nblk(c->nelems), kBlock, 0, c->st>>>(c->d_nodes, c->d_tri, (int)c->nnodes, (int)c->nelems,
                                                        (double)c->inor, c->d_surf, flag);
  IB3D_CUDA(c, cudaGetLastError());
  return IB3D_OK;
}

// One round of the level search: l = 1 + max level of the sources. Levels only grow, so a
// round that reads another op's newer level is as good. ctl[0] becomes r + 1 when the round
// changed something.
__global__ void k_level_round(int n, const int* __restrict__ src, int* lvl, int r, int* ctl) {
  if (*ctl < r) return;   // the last round changed nothing
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int l = 0;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int e = src[8 * (size_t)q + s];
    if (e >= 0) l = max(l, ((volatile int*)lvl)[e] + 1);
  }
  if (l != lvl[q]) {
    lvl[q] = l;
    atomicMax(ctl, r + 1);
  }
}
// Ops per level; the last of `most` counts also takes what lies beyond. Counted per block
// first: nearly all ops are of one level, and one counter for all of them took 31 us.
__global__ void __launch_bounds__(kBlock) k_level_count(int n, const int* __restrict__ lvl, int most, int* cnt) {
  __shared__ int s[32];
  if (threadIdx.x < 32) s[threadIdx.x] = 0;
  __syncthreads();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) atomicAdd(&s[min(lvl[q], most - 1)], 1);
  __syncthreads();
  if (threadIdx.x < (unsigned)most && s[threadIdx.x]) atomicAdd(&cnt[threadIdx.x], s[threadIdx.x]);
}
struct LevelStart {
  int at[32];
};
// The ops of each level together, in no particular order: those of one level do not depend
// on one another.
__global__ void __launch_bounds__(kBlock) k_level_scatter(int n, const int* __restrict__ lvl, LevelStart start,
                                                          int* __restrict__ used, int* __restrict__ order) {
  __shared__ int s[32], at[32];
  if (threadIdx.x < 32) s[threadIdx.x] = 0;
  __syncthreads();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int l = q < n ? lvl[q] : 0;
  const int mine = q < n ? atomicAdd(&s[l], 1) : 0;
  __syncthreads();
  if (threadIdx.x < 32 && s[threadIdx.x]) at[threadIdx.x] = start.at[threadIdx.x] + atomicAdd(&used[threadIdx.x], s[threadIdx.x]);
  __syncthreads();
  if (q < n) order[at[l] + mine] = q;
}

namespace {
void free_sched(ForceSched& s) {
  cudaFree(s.lvl);
  cudaFree(s.order); cudaFree(s.rd_idx); cudaFree(s.rd_src); cudaFree(s.tgt); cudaFree(s.brk);
  cudaFree(s.fin); cudaFree(s.out);
  s = ForceSched{};
}

// Dependency levels (level = 1 + max level of the sources; sources precede the op in
// serial order) and the level-sorted op list, for a schedule in which some op reads
// another's value. The levels settle on the device in as many rounds as there are levels
// (a handful); a schedule that is still moving after kRounds, or has more than kMaxLevels,
// is sorted on the host (the copies and loops of that took 0.35 ms at 45,000 ops).
constexpr int kRounds = 8, kMaxLevels = 32;   // k_level_count and k_level_scatter hold 32
int build_levels_host(ib3d_ctx* c, ForceSched& s) {
  const int n = s.nops;
  std::vector<int> src((size_t)8 * n), lvl(n, 0);
  IB3D_CUDA(c, cudaMemcpyAsync(src.data(), s.rd_src, sizeof(int) * 8 * (size_t)n, cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  int maxl = -1;
  for (int q = 0; q < n; ++q) {
    int l = 0;
    for (int r = 0; r < 8; ++r) {
      const int sidx = src[8 * (size_t)q + r];
      if (sidx >= 0) l = std::max(l, lvl[sidx] + 1);
    }
    lvl[q] = l;
    maxl = std::max(maxl, l);
  }
  s.nlevels = maxl + 1;
  s.level_off.assign((size_t)s.nlevels + 1, 0);
  for (int q = 0; q < n; ++q) s.level_off[lvl[q] + 1]++;
  for (int l = 0; l < s.nlevels; ++l) s.level_off[l + 1] += s.level_off[l];
  std::vector<int> order(n), pos(s.level_off.begin(), s.level_off.end() - 1);
  for (int q = 0; q < n; ++q) order[pos[lvl[q]]++] = q;
  IB3D_CUDA(c, cudaMemcpyAsync(s.order, order.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  s.ordered = true;
  return IB3D_OK;
}

// ctl: [0] rounds that changed a level, [1..kMaxLevels] ops per level (the last one also
// counts what lies beyond)
int build_levels(ib3d_ctx* c, ForceSched& s) {
  const int n = s.nops;
  int* ctl = c->d_levels;
  IB3D_CUDA(c, cudaMemsetAsync(s.lvl, 0, sizeof(int) * (size_t)n, c->st));
  IB3D_CUDA(c, cudaMemsetAsync(ctl, 0, sizeof(int) * (2 * kMaxLevels + 1), c->st));
  for (int r = 0; r < kRounds; ++r) k_level_round<<<nblk(n), kBlock, 0, c->st>>>(n, s.rd_src, s.lvl, r, ctl);
  k_level_count<<<nblk(n), kBlock, 0, c->st>>>(n, s.lvl, kMaxLevels, ctl + 1);
  int h[kMaxLevels + 1];
  IB3D_CUDA(c, cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  if (h[0] >= kRounds || h[kMaxLevels] != 0) return build_levels_host(c, s);
  s.nlevels = 0;
  s.level_off.assign(1, 0);
  for (int l = 0; l < kMaxLevels && h[1 + l] > 0; ++l) {
    s.level_off.push_back(s.level_off.back() + h[1 + l]);
    ++s.nlevels;
  }
  LevelStart start{};
  for (int l = 0; l < s.nlevels; ++l) start.at[l] = s.level_off[l];
  k_level_scatter<<<nblk(n), kBlock, 0, c->st>>>(n, s.lvl, start, ctl + 1 + kMaxLevels, s.order);
  IB3D_CUDA(c, cudaGetLastError());
  s.ordered = true;
  return IB3D_OK;
}

// Room for nops ops, kept for the next search (a moving body searches every step), and a
// schedule of one level until build_levels finds more.
int alloc_sched(ib3d_ctx* c, ForceSched& s, int nops) {
  if (nops > s.cap || s.cap == 0) {
    const size_t n = (size_t)nops + (size_t)nops / 8 + 64;
    free_sched(s);
    IB3D_CUDA(c, cudaMalloc(&s.order, sizeof(int) * n));
    IB3D_CUDA(c, cudaMalloc(&s.lvl, sizeof(int) * n));
    IB3D_CUDA(c, cudaMalloc(&s.rd_idx, sizeof(int) * 8 * n));
    IB3D_CUDA(c, cudaMalloc(&s.rd_src, sizeof(int) * 8 * n));
    IB3D_CUDA(c, cudaMalloc(&s.tgt, sizeof(int) * n));
    IB3D_CUDA(c, cudaMalloc(&s.brk, sizeof(int) * 3 * n));
    IB3D_CUDA(c, cudaMalloc(&s.fin, n));
    IB3D_CUDA(c, cudaMalloc(&s.out, sizeof(double) * n));
    s.cap = (int)n;
  }
  s.nops = nops;
  s.ordered = false;
  s.nlevels = nops > 0 ? 1 : 0;
  s.level_off.assign({0, nops});
  return IB3D_OK;
}
}  // namespace

void free_ib(ib3d_ctx* c) {
  free_sched(c->fv);
  free_sched(c->fp);
}

namespace {
// Scratch of at least `n` long longs in c->d_scan (counts at 0..7, block offsets from 8).
int ensure_scan(ib3d_ctx* c, size_t n) {
  if (n + 9 > c->scan_cap) {
    cudaFree(c->d_scan);
    c->d_scan = nullptr;
    c->scan_cap = 0;
    IB3D_CUDA(c, cudaMalloc(&c->d_scan, sizeof(long long) * (n + 64)));
    c->scan_cap = n + 64;
  }
  return IB3D_OK;
}
// Nearest elements of the box's cells, room kept for the next search.
int ensure_minel(ib3d_ctx* c, size_t nbox) {
  if (nbox > c->minel_cap) {
    cudaFree(c->d_minel);
    c->d_minel = nullptr;
    c->minel_cap = 0;
    const size_t n = nbox + nbox / 4;
    IB3D_CUDA(c, cudaMalloc(&c->d_minel, sizeof(int) * n));
    c->minel_cap = n;
  }
  return IB3D_OK;
}
// The IB list with its elements and distances, room kept for the next search.
int ensure_ib(ib3d_ctx* c, size_t nib) {
  if (nib > c->ib_cap || c->ib_cap == 0) {
    cudaFree(c->d_iblist); cudaFree(c->d_nelp); cudaFree(c->d_nd);
    c->d_iblist = nullptr; c->d_nelp = nullptr; c->d_nd = nullptr;
    c->ib_cap = 0;
    const size_t n = nib + nib / 8 + 64;
    IB3D_CUDA(c, cudaMalloc(&c->d_iblist, sizeof(int) * 3 * n));
    IB3D_CUDA(c, cudaMalloc(&c->d_nelp, sizeof(int) * n));
    IB3D_CUDA(c, cudaMalloc(&c->d_nd, sizeof(double) * 7 * n));
    c->ib_cap = n;
  }
  return IB3D_OK;
}
// The FP32 centroids and their groups for k_tagging, from the surface as it is now.
int group_centroids(ib3d_ctx* c) {
  const int ne = (int)c->nelems, gs = group_size(ne), ng = (ne + gs - 1) / gs;
  IB3D_CUDA(c, cudaMemsetAsync(c->d_c32_max, 0, sizeof(unsigned), c->st));
  k_centroid_groups<<<(ng + 7) / 8, 256, 0, c->st>>>(c->d_surf, ne, c->d_c32, c->d_c32_max);
  IB3D_CUDA(c, cudaGetLastError());
  return IB3D_OK;
}
int finish_search(ib3d_ctx* c, int bi0, int bj0, int bk0, int bni, int bnj, int bnk);
}  // namespace

int run_search(ib3d_ctx* c) {
  const Dims& d = c->d;
  const int bi0 = (int)c->box[0], bj0 = (int)c->box[2], bk0 = (int)c->box[4];
  const int bni = (int)(c->box[1] - c->box[0] + 1), bnj = (int)(c->box[3] - c->box[2] + 1),
            bnk = (int)(c->box[5] - c->box[4] + 1);
  const unsigned nbox = (unsigned)bni * bnj * bnk;
  const int ne = (int)c->nelems;
  // fresh flags and maps
  IB3D_CUDA(c, cudaMemsetAsync(c->cell, 0, (size_t)d.n3, c->st));
  if (int rc = ensure_minel(c, nbox)) return rc;
  if (int rc = group_centroids(c)) return rc;
  k_tagging<<<nblk(4ll * nbox), kBlock, 0, c->st>>>(d, c->g, c->d_surf, ne, c->d_c32, c->d_c32_max, bi0, bj0, bk0, bni, bnj, bnk, nullptr, 0,
                                               c->cell, c->d_minel);
  IB3D_CUDA(c, cudaGetLastError());
  return finish_search(c, bi0, bj0, bk0, bni, bnj, bnk);
}

// selectiveRetagging (subSearch.f90:327-512): the tagging test on the 6x6x6
// neighbourhood of every cell of the current IB list, every other cell keeping its
// flag; then the counts, the IB list, the normal distances and the ghost-point
// schedules as after a full search. The neighbourhoods' cells are marked in a mask
// over their bounding box (clipped to the interior), compacted into a list, and only
// those are tagged.
int run_selective_retag(ib3d_ctx* c) {
  const Dims& d = c->d;
  const int nib = c->nib, ne = (int)c->nelems;
  int* dbound = reinterpret_cast<int*>(c->d_scan);
  const int init[6] = {0x7fffffff, -0x7fffffff, 0x7fffffff, -0x7fffffff, 0x7fffffff, -0x7fffffff};
  IB3D_CUDA(c, cudaMemcpyAsync(dbound, init, sizeof(init), cudaMemcpyHostToDevice, c->st));
  k_ib_bounds<<<std::min(nblk(nib), 64u), kBlock, 0, c->st>>>(c->d_iblist, nib, dbound);
  int hb[6];
  IB3D_CUDA(c, cudaMemcpyAsync(hb, dbound, sizeof(hb), cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  const int bi0 = std::max(hb[0] - 2, 2), bi1 = std::min(hb[1] + 3, d.nx + 1);
  const int bj0 = std::max(hb[2] - 2, 2), bj1 = std::min(hb[3] + 3, d.ny + 1);
  const int bk0 = std::max(hb[4] - 2, 2), bk1 = std::min(hb[5] + 3, d.nz + 1);
  const int bni = bi1 - bi0 + 1, bnj = bj1 - bj0 + 1, bnk = bk1 - bk0 + 1;
  const unsigned nbox = (unsigned)bni * bnj * bnk;
  if (int rc = ensure_minel(c, nbox)) return rc;
  IB3D_CUDA(c, cudaMemsetAsync(c->d_minel, 0, sizeof(int) * (size_t)nbox, c->st));
  if ((size_t)nbox > c->retag_cap) {
    cudaFree(c->d_retag_mask);
    cudaFree(c->d_retag_list);
    c->d_retag_mask = nullptr;
    c->d_retag_list = nullptr;
    c->retag_cap = 0;
    const size_t n = (size_t)nbox + (size_t)nbox / 4;
    IB3D_CUDA(c, cudaMalloc(&c->d_retag_mask, n));
    IB3D_CUDA(c, cudaMalloc(&c->d_retag_list, 3 * sizeof(int) * n));
    c->retag_cap = n;
  }
  IB3D_CUDA(c, cudaMemsetAsync(c->d_retag_mask, 0, nbox, c->st));
  k_mark_neighbourhoods<<<nblk(216ll * nib), kBlock, 0, c->st>>>(c->d_iblist, nib, bi0, bj0, bk0, bni, bnj, bnk,
                                                                  c->d_retag_mask);
  const unsigned nb = nblk(nbox);
  if (int rc = ensure_scan(c, nb)) return rc;
  long long* boff = c->d_scan + 8;
  k_mask_blockcount<<<nb, kBlock, 0, c->st>>>(c->d_retag_mask, nbox, boff);
  k_exclusive_scan<<<1, 1024, 0, c->st>>>(boff, (int)nb, c->d_scan);
  long long nlist = 0;
  IB3D_CUDA(c, cudaMemcpyAsync(&nlist, c->d_scan, sizeof(long long), cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  // the list is sized for the whole box: the three index blocks start nlist apart
  k_mask_scatter<<<nb, kBlock, 0, c->st>>>(c->d_retag_mask, nbox, bi0, bj0, bk0, bni, bnj, boff, (int)nlist,
                                           c->d_retag_list);
  if (int rc = group_centroids(c)) return rc;
  if (nlist > 0)
    k_tagging<<<nblk(4ll * nlist), kBlock, 0, c->st>>>(d, c->g, c->d_surf, ne, c->d_c32, c->d_c32_max, bi0, bj0, bk0, bni, bnj, bnk,
                                                 c->d_retag_list, (int)nlist, c->cell, c->d_minel);
  IB3D_CUDA(c, cudaGetLastError());
  c->retagged = nlist;
  return finish_search(c, bi0, bj0, bk0, bni, bnj, bnk);
}

namespace {
// The part of the search after the flags are set: counts, the lexicographic IB list
// over the box (every IB cell lies in it), the normal distances and the ghost-point
// schedules.
int finish_search(ib3d_ctx* c, int bi0, int bj0, int bk0, int bni, int bnj, int bnk) {
  const Dims& d = c->d;
  const unsigned nbox = (unsigned)bni * bnj * bnk;
  const int ne = (int)c->nelems;
  const unsigned nb = nblk(nbox);
  if (int rc = ensure_scan(c, nb)) return rc;
  IB3D_CUDA(c, cudaMemsetAsync(c->ibmap, 0xff, sizeof(int) * (size_t)d.n3, c->st));
  // counts
  unsigned long long* dcount = reinterpret_cast<unsigned long long*>(c->d_scan);
  IB3D_CUDA(c, cudaMemsetAsync(dcount, 0, 5 * sizeof(unsigned long long), c->st));
  k_count<<<std::min(nblk((long long)d.nx * d.ny * d.nz), 8u * (unsigned)c->nsm), kBlock, 0, c->st>>>(d, c->cell, dcount);
  unsigned long long hc[5];
  IB3D_CUDA(c, cudaMemcpyAsync(hc, dcount, sizeof(hc), cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  for (int q = 0; q < 5; ++q) c->counts[q] = (long long)hc[q];
  c->nib = (int)hc[2];
  const int nib = c->nib;
  // compaction of the IB cells
  if (int rc = ensure_ib(c, (size_t)nib)) return rc;
  long long* boff = c->d_scan + 8;
  k_ib_blockcount<<<nb, kBlock, 0, c->st>>>(d, c->cell, bi0, bj0, bk0, bni, bnj, nbox, boff);
  k_exclusive_scan<<<1, 1024, 0, c->st>>>(boff, (int)nb, c->d_scan);
  k_ib_scatter<<<nb, kBlock, 0, c->st>>>(d, c->cell, bi0, bj0, bk0, bni, bnj, nbox, boff, nib, c->d_iblist);
  if (nib > 0)
    k_normdist<<<nblk(nib), kBlock, 0, c->st>>>(d, c->g, c->d_surf, ne, c->d_iblist, nib, c->d_minel, bi0, bj0,
                                                bk0, bni, bnj, c->d_nelp, c->d_nd, c->ibmap);
  IB3D_CUDA(c, cudaGetLastError());
  // ghost-point schedules
  IB3D_CUDA(c, cudaMemsetAsync(c->d_flag, 0, 3 * sizeof(int), c->st));
  int rc = alloc_sched(c, c->fv, 6 * nib);
  if (rc) return rc;
  rc = alloc_sched(c, c->fp, nib);
  if (rc) return rc;
  if (nib > 0) {
    k_sched_vel<<<nblk(6ll * nib), kBlock, 0, c->st>>>(d, c->g, c->d_iblist, c->d_nelp, c->d_nd, c->d_surf, nib, ne,
                                                       c->ibmap, c->fv.brk, c->fv.rd_idx, c->fv.rd_src, c->fv.tgt,
                                                       c->fv.fin, c->d_flag, c->d_flag + 1);
    k_sched_p<<<nblk(nib), kBlock, 0, c->st>>>(d, c->g, c->d_iblist, c->d_nelp, c->d_nd, c->d_surf, nib, ne,
                                               c->ibmap, c->fp.brk, c->fp.rd_idx, c->fp.rd_src, c->fp.tgt, c->fp.fin,
                                               c->d_flag, c->d_flag + 2);
    IB3D_CUDA(c, cudaGetLastError());
  }
  int flag[3] = {0, 0, 0};   // a probe off the grid; ops of the velocity, of the pressure depend on one another
  IB3D_CUDA(c, cudaMemcpyAsync(flag, c->d_flag, sizeof(flag), cudaMemcpyDeviceToHost, c->st));
  IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  if (flag[1] && (rc = build_levels(c, c->fv))) return rc;
  if (flag[2] && (rc = build_levels(c, c->fp))) return rc;
  c->have_scache = false;
  if (flag[0]) {
    c->err = "ib3d_search: a ghost-point probe fell outside the grid";
    return IB3D_ERR_PROBE;
  }
  return IB3D_OK;
}
}  // namespace

int run_velocity_forcing(ib3d_ctx* c) {
  PhaseScope ps(c, PH_FORCING);
  ForceSched& s = c->fv;
  c->launches += s.nlevels + (s.nops > 0 ? 1 : 0);
  for (int l = 0; l < s.nlevels; ++l) {
    const int off = s.level_off[l], cnt = s.level_off[l + 1] - off;
    if (cnt <= 0) continue;
    k_force_vel<<<nblk(cnt, 64), 64, 0, c->st>>>(c->g, s.ordered ? s.order : nullptr, off, cnt, c->d_iblist, c->d_nelp, c->d_nd, c->d_surf,
                                                 c->nib, (int)c->nelems, s.brk, s.rd_idx, s.rd_src, c->ut, c->vt,
                                                 c->wt, c->motion, s.out);
  }
  if (s.nops > 0)
    k_force_scatter<<<nblk(s.nops), kBlock, 0, c->st>>>(s.fin, s.nops, s.tgt, s.out, 1, c->ut, c->vt,
                                                          c->wt);
  IB3D_CUDA(c, cudaGetLastError());
  return IB3D_OK;
}

int run_pressure_forcing(ib3d_ctx* c) {
  PhaseScope ps(c, PH_FORCING);
  ForceSched& s = c->fp;
  for (int q = 0; q < 3; ++q) c->motion.acc[q] = -(c->motion.vel[q] - c->bprev[q]) / c->prm.deltat;   // :20
  c->launches += s.nlevels + (s.nops > 0 ? 1 : 0);
  for (int l = 0; l < s.nlevels; ++l) {
    const int off = s.level_off[l], cnt = s.level_off[l + 1] - off;
    if (cnt <= 0) continue;
    k_force_p<<<nblk(cnt, 64), 64, 0, c->st>>>(c->g, s.ordered ? s.order : nullptr, off, cnt, c->d_iblist, c->d_nelp, c->d_nd, c->d_surf,
                                               c->nib, (int)c->nelems, s.brk, s.rd_idx, s.rd_src, c->p, c->motion,
                                               s.out);
  }
  if (s.nops > 0)
    k_force_scatter<<<nblk(s.nops), kBlock, 0, c->st>>>(s.fin, s.nops, s.tgt, s.out, 0, c->p, nullptr,
                                                          nullptr);
  IB3D_CUDA(c, cudaGetLastError());
  return IB3D_OK;
}

int run_stress(ib3d_ctx* c, int first, double coef[4]) {
  const int ne = (int)c->nelems;
  const int do_first = (first || !c->have_scache) ? 1 : 0;
  if (do_first) IB3D_CUDA(c, cudaMemsetAsync(c->d_flag, 0, sizeof(int), c->st));
  PhaseScope ps(c, PH_STRESS);
  c->launches += 2;
  k_stress_elem<<<nblk(4ll * ne, 64), 64, 0, c->st>>>(c->d, c->g, c->d_surf, ne, do_first, c->d_scache, c->ut, c->vt,
                                                      c->wt, c->p, 1.0 / c->prm.re, c->d_contrib, c->d_flag);
  if (c->prm.precision == IB3D_PREC_FP64) k_stress_sum<<<1, kSumThreads, 0, c->st>>>(c->d_contrib, ne, c->d_coef);
  else k_stress_sum_tree<<<7, kTreeThreads, 0, c->st>>>(c->d_contrib, ne, c->d_coef);
  IB3D_CUDA(c, cudaGetLastError());
  if (do_first) {
    int flag = 0;
    IB3D_CUDA(c, cudaMemcpyAsync(&flag, c->d_flag, sizeof(int), cudaMemcpyDeviceToHost, c->st));
    IB3D_CUDA(c, cudaStreamSynchronize(c->st));
    if (flag) {
      c->err = "ib3d_stress: a drag probe fell outside the grid";
      return IB3D_ERR_PROBE;
    }
    c->have_scache = true;
  }
  if (coef) {
    IB3D_CUDA(c, cudaMemcpyAsync(coef, c->d_coef, 4 * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    IB3D_CUDA(c, cudaStreamSynchronize(c->st));
  }
  return IB3D_OK;
}

}  // namespace ib3d
