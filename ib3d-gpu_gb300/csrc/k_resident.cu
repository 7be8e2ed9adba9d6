// Red-black sweeps with the unknowns kept in shared memory: one cooperative launch runs a
// whole batch of sweeps.
//
// A colour pass of the launch-per-pass kernels takes 2.5-5 us on a grid of 0.1-2 M cells
// whatever its arithmetic: the launch, the drain of the last pass and one chain of L2
// latencies per plane. Here every block keeps by x bz whole rows of the grid in shared
// memory for all sweeps -- the unknowns of both colours with one ghost row around, and
// the right-hand side -- and only the rows at a block's edges travel.
//
// Exchange. After a pass a block publishes the updated colour's values of its edge rows to
// the up to four neighbouring blocks through global memory (L2), each value paired in one
// 64-bit word with the number of the pass, and polls its neighbours' words until they carry
// the same number. A word is stored and loaded whole, so the data needs no fence and no
// separate flag, and a pass costs one L2 store and about one load latency instead of a
// fence, a flag and two loads. Each pass rewrites every word with the next number of its
// colour, so an old word never passes for a new one. A word is not overwritten before its
// reader has it: a block enters pass p + 2 only after it has received the words of pass
// p + 1 from every neighbour, which that neighbour published after all its threads had
// read pass p (one block barrier ends each pass).
//
// The blocks wait on one another, so the launch is cooperative (all blocks resident, and started
// together: a solve beside a kernel that held 100 SMs for 1.5 s began when it had ended). A
// wait gives up after a bounded number of polls, or when another block has given up: the block
// sets the error flag and returns without storing. A block whose last waits had already ended
// stores its rows all the same, so the array that the launch writes is then part old, part new,
// and the solve ends with an error. The words left behind carry numbers that no later launch
// waits for. The kernels run on one stream at a time per exchange buffer.
//
// Compiled with -fmad=false: the FP64 kernel keeps the reference's rounding.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "resident.cuh"
#include "sor32_update.cuh"

namespace ib3d {

namespace {

typedef unsigned long long u64;

constexpr int kHalo = 4;                  // received items per thread, at most
constexpr int kMaxThreads = 512;
constexpr size_t kSmemCap = 227 * 1024 - 1024;

// The limit belongs to the kernel, not to a context: always the largest plan's, so that no
// thread's launch meets another's smaller one.
cudaError_t allow_smem(const void* kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
}

__device__ __forceinline__ void st_pair(u64* p, u64 a, u64 b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" :: "l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_pair(const u64* p, u64& a, u64& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ int ld_flag(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld4s(const float* p) { return *reinterpret_cast<const float4*>(p); }

__device__ __forceinline__ u64 tagged(unsigned bits, unsigned seq) { return ((u64)seq << 32) | bits; }

// The rows of this block: [j0, j0 + nyb) x [k0, k0 + nzb).
struct Span {
  int jb, kb, j0, k0, nyb, nzb;
};
__device__ __forceinline__ Span block_span(const Dims& d, int gy, int gz) {
  Span s;
  s.jb = (int)blockIdx.x % gy;
  s.kb = (int)blockIdx.x / gy;
  const int a = s.jb * d.ny / gy, b = (s.jb + 1) * d.ny / gy;
  const int c = s.kb * d.nz / gz, e = (s.kb + 1) * d.nz / gz;
  s.j0 = 2 + a; s.nyb = b - a;
  s.k0 = 2 + c; s.nzb = e - c;
  return s;
}

// Edge rows of a block in the exchange buffer: low y edge (row kk), high y edge, low z edge
// (row jj), high z edge.
__device__ __forceinline__ int edge_ylo(int kk) { return kk; }
__device__ __forceinline__ int edge_yhi(int bz, int kk) { return bz + kk; }
__device__ __forceinline__ int edge_zlo(int bz, int jj) { return 2 * bz + jj; }
__device__ __forceinline__ int edge_zhi(int by, int bz, int jj) { return 2 * bz + by + jj; }

// Ghost row h of a block (0 <= h < 2 nzb + 2 nyb): its place (kk, jj) around the block's
// rows, and the neighbouring block and edge row it comes from; false at the domain's edge,
// whose ghost row has no writer.
__device__ __forceinline__ bool ghost_row(const Span& s, int gy, int gz, int by, int bz, int h, int& kk, int& jj,
                                          int& nb, int& er) {
  const int me = s.kb * gy + s.jb;
  if (h < s.nzb) {
    kk = h; jj = -1; nb = me - 1; er = edge_yhi(bz, kk);
    return s.jb > 0;
  }
  h -= s.nzb;
  if (h < s.nzb) {
    kk = h; jj = s.nyb; nb = me + 1; er = edge_ylo(kk);
    return s.jb + 1 < gy;
  }
  h -= s.nzb;
  if (h < s.nyb) {
    kk = -1; jj = h; nb = me - gy; er = edge_zhi(by, bz, jj);
    return s.kb > 0;
  }
  kk = s.nzb; jj = h - s.nyb; nb = me + gy; er = edge_zlo(bz, jj);
  return s.kb + 1 < gz;
}

}  // namespace

// FP32 sweeps (the inner solve of the defect correction) on the colour-packed rows of
// k_sor32.cu. Per cell the operations and their order are update4's, so the results have
// the bits of the launch-per-pass kernels.
//
// A thread owns one float4 group of a row position over zl consecutive planes and marches
// through them: the other colour's values of a plane serve as the lower neighbour, the
// centre and the upper neighbour of three planes, so a plane costs five 16-byte
// shared-memory loads (next plane, two y neighbours, right-hand side, own value) and a
// store instead of ten accesses, and the x coefficients of both row phases stay in
// registers. Threads beyond the owners only receive ghost rows. NH: received groups per
// thread. (Both colours' values in registers as well would halve the accesses, but from
// four planes on the registers spill: 128^3 5.6 against 5.0 us per sweep.)
template <int NH>
__global__ void __launch_bounds__(kMaxThreads, 1) k_resident32(Resident32 A) {
  extern __shared__ __align__(16) float sm[];
  const Dims& d = A.d;
  const int nq = row_groups(d.nx), Lr = 4 * nq + 8;
  const int plane = (A.by + 2) * Lr, all = (A.bz + 2) * plane;
  const Span s = block_span(d, A.gy, A.gz);
  const int nt = blockDim.x, t = threadIdx.x, lane = t & 31;
  const int planeR = A.by * 4 * nq, allR = A.bz * planeR;
  float* E = sm;                                       // [2][all]
  float* R = E + 2 * all;                              // [2][allR]
  float4* Z = reinterpret_cast<float4*>(R + 2 * allR); // [bz]: the plane's three z coefficients
  for (int n = t; n < 2 * all; n += nt) E[n] = 0.f;
  for (int n = t; n < s.nzb; n += nt)
    Z[n] = make_float4(A.az[0][s.k0 + n - 1], A.az[1][s.k0 + n - 1], A.az[2][s.k0 + n - 1], 0.f);
  const int cols = s.nyb * nq;
  const int chunk = t / cols, col = t - chunk * cols, jj = col / nq, q = col - jj * nq;
  const int kk0 = chunk * A.zl, len = min(A.zl, s.nzb - kk0);   // this thread's planes kk0 .. kk0 + len - 1
  const bool own = len > 0;
  const int ER = 2 * (A.by + A.bz);                    // edge rows per block and colour
  const int cstride = ER * 4 * nq;                     // exchange words per block and colour
  u64* mine = A.xch + (size_t)blockIdx.x * 2 * cstride;
  // this thread's column: place in E and R, y edge (0 none, 1 low, 2 high), coefficients
  const int off0 = (jj + 1) * Lr + 4 * q + 4, offR = jj * 4 * nq + 4 * q;
  const int yedge = !own ? 0 : jj == 0 && s.jb > 0 ? 1 : jj == s.nyb - 1 && s.jb + 1 < A.gy ? 2 : 0;
  // f0: does the row at plane kk0 start (i = 2) with red? Phase arrays: [0] the phase of
  // red at even steps of the march (and of black at odd ones), [1] the other
  const bool f0 = ((s.j0 + jj + s.k0 + kk0) & 1) == 1;
  float4 x0[2], x1[2], x2[2];
  float ay0 = 0.f, ay1 = 0.f, ay2 = 0.f;
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int sp = (f == 0) == f0 ? 0 : 1;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    x0[f] = own ? A.axp[sp][0][q] : z4;
    x1[f] = own ? A.axp[sp][1][q] : z4;
    x2[f] = own ? A.axp[sp][2][q] : z4;
  }
  if (own) {
    ay0 = A.ay[0][s.j0 + jj - 1];
    ay1 = A.ay[1][s.j0 + jj - 1];
    ay2 = A.ay[2][s.j0 + jj - 1];
    for (int c = 0; c < 2; ++c)
      for (int kk = kk0; kk < kk0 + len; ++kk)
        *reinterpret_cast<float4*>(R + c * allR + kk * planeR + offR) = __ldg(reinterpret_cast<const float4*>(
            A.r[c] + (size_t)(s.k0 + kk - 2) * A.ps + (size_t)(s.j0 + jj - 2) * A.rs + 4 * q));
  }
  const u64* hsrc[NH];
  int hdst[NH];
  const int ghosts = 2 * (s.nyb + s.nzb) * nq;
  bool wait_any = false;
#pragma unroll
  for (int n = 0; n < NH; ++n) {
    hdst[n] = -1;
    hsrc[n] = nullptr;
    const int h = nt - 1 - t + n * nt;
    if (h < ghosts) {
      const int row = h / nq, g = h - row * nq;
      int kk, gj, nb, er;
      if (ghost_row(s, A.gy, A.gz, A.by, A.bz, row, kk, gj, nb, er)) {
        hdst[n] = (kk + 1) * plane + (gj + 1) * Lr + 4 * g + 4;
        hsrc[n] = A.xch + (size_t)nb * 2 * cstride + (size_t)(er * nq + g) * 4;
        wait_any = true;
      }
    }
  }
  __syncthreads();
  bool fail = false;
  for (int sweep = 0; sweep < A.nsweeps; ++sweep) {
    float w = A.om, w1 = A.om1;
    if (sweep < A.nsmooth) {
      w = 1.0f; w1 = 0.0f;
    } else if (sweep < A.nsmooth + A.nramp) {
      const double wr = 1.0 + (double)(sweep - A.nsmooth + 1) / (A.nramp + 1) * (A.wi - 1.0);
      w = (float)wr;
      w1 = (float)(1.0 - wr);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned seq = A.seq0 + 2u * (unsigned)sweep + (unsigned)c + 1u;
      if (__any_sync(0xffffffffu, own)) {
        const float* o = E + (1 - c) * all + (own ? kk0 + 1 : 0) * plane + off0;
        float* p = E + c * all + (own ? kk0 + 1 : 0) * plane + off0;
        const float* r = R + c * allR + (own ? kk0 : 0) * planeR + offR;
        float4 ob = ld4s(o - (own ? plane : 0)), ox = ld4s(o);
        for (int u2 = 0; u2 < A.zl; u2 += 2)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int u = u2 + h;
            if (u >= A.zl) break;
            float left = __shfl_up_sync(0xffffffffu, ox.w, 1), right = __shfl_down_sync(0xffffffffu, ox.x, 1);
            if (u < len) {
              if (lane == 0 || q == 0) left = o[-1];
              if (lane == 31 || q == nq - 1) right = o[4];
              const float4 s4 = ld4s(o - Lr), n4 = ld4s(o + Lr), t4 = ld4s(o + plane), r4 = ld4s(r), e4 = ld4s(p);
              const float4 z = Z[kk0 + u];
              const bool first = f0 == (((c + h) & 1) == 0);   // the row starts with the updated colour
              const float x[5] = {first ? left : ox.x, first ? ox.x : ox.y, first ? ox.y : ox.z, first ? ox.z : ox.w,
                                  first ? ox.w : right};
              const float rv[4] = {r4.x, r4.y, r4.z, r4.w}, sv[4] = {s4.x, s4.y, s4.z, s4.w};
              const float nv[4] = {n4.x, n4.y, n4.z, n4.w}, bv[4] = {ob.x, ob.y, ob.z, ob.w};
              const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
              float ev[4] = {e4.x, e4.y, e4.z, e4.w};
              update4(rv, ev, x, sv, nv, bv, tv, x0[(c + h) & 1], x1[(c + h) & 1], x2[(c + h) & 1], ay0, ay1, ay2, z.x,
                      z.y, z.z, w, w1);
              *reinterpret_cast<float4*>(p) = make_float4(ev[0], ev[1], ev[2], ev[3]);
              const int kk = kk0 + u;
              const int ze = kk == 0 && s.kb > 0 ? edge_zlo(A.bz, jj)
                             : kk == s.nzb - 1 && s.kb + 1 < A.gz ? edge_zhi(A.by, A.bz, jj) : -1;
              if (yedge != 0 || ze >= 0) {
                const u64 v0 = tagged(__float_as_uint(ev[0]), seq), v1 = tagged(__float_as_uint(ev[1]), seq);
                const u64 v2 = tagged(__float_as_uint(ev[2]), seq), v3 = tagged(__float_as_uint(ev[3]), seq);
                if (yedge != 0) {
                  u64* dst = mine + c * cstride + ((yedge == 1 ? edge_ylo(kk) : edge_yhi(A.bz, kk)) * nq + q) * 4;
                  st_pair(dst, v0, v1);
                  st_pair(dst + 2, v2, v3);
                }
                if (ze >= 0) {
                  u64* dst = mine + c * cstride + (ze * nq + q) * 4;
                  st_pair(dst, v0, v1);
                  st_pair(dst + 2, v2, v3);
                }
              }
              ob = ox;
              ox = t4;
              o += plane;
              p += plane;
              r += planeR;
            }
          }
      }
      if (wait_any) {
        unsigned pend = 0;
#pragma unroll
        for (int n = 0; n < NH; ++n) pend |= hdst[n] >= 0 ? 1u << n : 0u;
        for (int it = 0; pend != 0; ++it) {
          u64 v[NH][4];
#pragma unroll
          for (int n = 0; n < NH; ++n)
            if (pend >> n & 1) {
              ld_pair(hsrc[n] + c * cstride, v[n][0], v[n][1]);
              ld_pair(hsrc[n] + c * cstride + 2, v[n][2], v[n][3]);
            }
#pragma unroll
          for (int n = 0; n < NH; ++n)
            if (pend >> n & 1) {
              if ((unsigned)(v[n][0] >> 32) == seq + A.skew && (unsigned)(v[n][1] >> 32) == seq + A.skew &&
                  (unsigned)(v[n][2] >> 32) == seq + A.skew && (unsigned)(v[n][3] >> 32) == seq + A.skew) {
                *reinterpret_cast<float4*>(E + c * all + hdst[n]) =
                    make_float4(__uint_as_float((unsigned)v[n][0]), __uint_as_float((unsigned)v[n][1]),
                                __uint_as_float((unsigned)v[n][2]), __uint_as_float((unsigned)v[n][3]));
                pend &= ~(1u << n);
              }
            }
          if (pend != 0 && (it & 255) == 255 && (it > A.polls || ld_flag(A.err) != 0)) {
            fail = true;
            break;
          }
        }
      }
      if (__syncthreads_or(fail)) {
        if (t == 0) atomicExch(A.err, 1);
        return;
      }
    }
  }
  // pc += e (FP64 accumulation of the FP32 correction)
  if (own)
    for (int kk = kk0; kk < kk0 + len; ++kk) {
      const int j = s.j0 + jj, k = s.k0 + kk;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int i0 = ((c == 0) == (((j + k) & 1) == 1) ? 2 : 3) + 8 * q;
        double* p = A.pc + d.at(i0, j, k);
        const float* v = E + c * all + (kk + 1) * plane + off0;
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (v[m] != 0.0f && i0 + 2 * m <= d.nx + 1) p[2 * m] = p[2 * m] + (double)v[m];
      }
    }
}

// FP64 sweeps of the plain path (REDBLACKSOR, subPcorVcor.f90:148-212), one cell of a
// colour per item; both colours' pc of the block's rows, the ghost rows and the x ghost
// cells in shared memory, and b/dt and what the division needs per cell beside them (in
// registers they spilled).
//
// EXACT: the reference's arithmetic. The kernel is bound by the FP64 pipe (1.65 operations
// per clock and SM), and the division by the diagonal was the largest single item of
// k_sor64 (about 8.6 of its 27 operations a cell). The diagonal of a cell never changes
// within a solve, so the division runs as four fused operations from its precomputed
// reciprocal (div_known) with the same rounded quotient.
// Otherwise the fast plain form (IB3D_PREC_FP64_FAST), k_sor64_fast's operations.
//
// check == 0: every sweep's largest |pc_new - pc_old| goes to errs[sweep]; else every
// check-th sweep's largest |b/dt - A pc| (k_residual64's or k_residual_fast's operations).
// The host applies the stopping test afterwards and, when it stops inside the batch, runs
// the batch again from its unchanged input up to the stopping sweep.
template <bool EXACT>
__global__ void __launch_bounds__(kMaxThreads, 1) k_resident64(Resident64 A) {
  extern __shared__ __align__(16) double smd[];
  const Dims& d = A.d;
  const int nh = (d.nx + 1) >> 1, Ld = nh + 2;         // entry m of a row at m + 1, m = -1 .. nh
  const int plane = (A.by + 2) * Ld, all = (A.bz + 2) * plane, allB = A.by * A.bz * nh;
  const Span s = block_span(d, A.gy, A.gz);
  const int nt = blockDim.x, t = threadIdx.x;
  double* E = smd;                    // [2][all]
  double* B = E + 2 * all;            // [2][allB]
  double* X = B + 2 * allB;           // [3][nx + 1]
  double* Y = X + 3 * (d.nx + 1);     // [3][by]
  double* Z = Y + 3 * A.by;           // [3][bz]
  double* zh = Z + 3 * A.bz;          // [2][allB] EXACT: the diagonal's reciprocal, else omega / diagonal
  double* zl = zh + 2 * allB;         // [2][allB] EXACT: the rest of the reciprocal
  double* dg = zl + 2 * allB;         // [2][allB] EXACT: the diagonal
  // per item: kk << 22 | jj << 12 | m, and bits 30 + c where its cell of colour c is fluid
  unsigned* pos = reinterpret_cast<unsigned*>(EXACT ? dg + 2 * allB : zl);
  for (int e = t; e < 3 * d.nx; e += nt) X[(e / d.nx) * (d.nx + 1) + e % d.nx + 1] = A.ax[e / d.nx][e % d.nx + 1];
  for (int e = t; e < 3 * s.nyb; e += nt) Y[(e / s.nyb) * A.by + e % s.nyb] = A.ay[e / s.nyb][s.j0 + e % s.nyb - 1];
  for (int e = t; e < 3 * s.nzb; e += nt) Z[(e / s.nzb) * A.bz + e % s.nzb] = A.az[e / s.nzb][s.k0 + e % s.nzb - 1];
  // pc of the rows j0-1 .. j0+nyb, planes k0-1 .. k0+nzb, ghost cells included
  const int rows = (s.nyb + 2) * (s.nzb + 2);
  for (int e = t; e < rows * d.NX2; e += nt) {
    const int row = e / d.NX2, i = e - row * d.NX2 + 1, kk = row / (s.nyb + 2) - 1, jj = row % (s.nyb + 2) - 1;
    const int j = s.j0 + jj, k = s.k0 + kk;
    const int c = ((i + j + k) & 1) ? 0 : 1;
    const int m = (i & 1) ? (i - 3) / 2 : (i - 2) / 2;   // rows start with even i in one colour, odd i in the other
    E[c * all + (kk + 1) * plane + (jj + 1) * Ld + m + 1] = A.pc_in[d.at(i, j, k)];
  }
  const int items = s.nyb * s.nzb * nh;
  const int ER = 2 * (A.by + A.bz), cstride = ER * 2 * nh;   // a value takes two words
  u64* mine = A.xch + (size_t)blockIdx.x * 2 * cstride;
  for (int it = t; it < items; it += nt) {
    const int row = it / nh, m = it - row * nh, kk = row / s.nyb, jj = row - kk * s.nyb;
    const int j = s.j0 + jj, k = s.k0 + kk;
    unsigned p = (unsigned)(kk << 22 | jj << 12 | m);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int i = ((c == 0) == (((j + k) & 1) == 1) ? 2 : 3) + 2 * m;
      if (i > d.nx + 1) continue;
      const long long o = d.at(i, j, k);
      if (A.cell[o] != 0) continue;
      const int q = c * allB + it;
      B[q] = A.bdt[o];
      const double diag = A.ax[1][i - 1] + A.ay[1][j - 1] + A.az[1][k - 1];
      const double r = (EXACT ? 1.0 : A.omega) / diag;
      zh[q] = r;
      if (EXACT) {
        dg[q] = diag;
        zl[q] = fma(-r, diag, 1.0) / diag;
      }
      if (EXACT || r != 0.0) p |= 1u << (30 + c);
    }
    pos[it] = p;
  }
  const u64* hsrc[kHalo];
  int hdst[kHalo];
  const int ghosts = 2 * (s.nyb + s.nzb) * nh;
#pragma unroll
  for (int n = 0; n < kHalo; ++n) {
    hdst[n] = -1;
    hsrc[n] = nullptr;
    const int h = nt - 1 - t + n * nt;
    if (h < ghosts) {
      const int row = h / nh, m = h - row * nh;
      int kk, jj, nb, er;
      if (ghost_row(s, A.gy, A.gz, A.by, A.bz, row, kk, jj, nb, er)) {
        hdst[n] = (kk + 1) * plane + (jj + 1) * Ld + m + 1;
        hsrc[n] = A.xch + (size_t)nb * 2 * cstride + (size_t)(er * nh + m) * 2;
      }
    }
  }
  __syncthreads();
  bool fail = false;
  u64 big = 0;                                         // largest update of the sweep
  for (int sweep = 0; sweep < A.nsweeps; ++sweep) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double* Eo = E + (1 - c) * all;
      double* Ec = E + c * all;
      const unsigned seq = A.seq0 + 2u * (unsigned)sweep + (unsigned)c + 1u;
      for (int it = t; it < items; it += nt) {
        const unsigned ps = pos[it];
        const int m = ps & 4095u, jj = ps >> 12 & 1023u, kk = ps >> 22 & 255u;
        const int off = (kk + 1) * plane + (jj + 1) * Ld + m + 1;
        const bool first = (c == 0) == (((s.j0 + jj + s.k0 + kk) & 1) == 1);
        double nw = Ec[off];
        if (ps >> (30 + c) & 1) {
          const double* o = Eo + off;
          const int i = (first ? 2 : 3) + 2 * m, q = c * allB + it;
          const double old = nw, bd = B[q];
          const double W = first ? o[-1] : o[0], Ea = first ? o[0] : o[1];
          const double a0 = X[i - 1], a2 = X[2 * (d.nx + 1) + i - 1];
          const double y0 = Y[jj], y2 = Y[2 * A.by + jj], z0 = Z[kk], z2 = Z[2 * A.bz + kk];
          if (EXACT) {
            const double num = bd - a0 * W - a2 * Ea - y0 * o[-Ld] - y2 * o[Ld] - z0 * o[-plane] - z2 * o[plane];
            const double gs = div_known(num, dg[q], zh[q], zl[q]);
            nw = A.om1 * old + A.omega * gs;
          } else {
            double num = fma(-a0, W, bd);
            num = fma(-a2, Ea, num);
            num = fma(-y0, o[-Ld], num);
            num = fma(-y2, o[Ld], num);
            num = fma(-z0, o[-plane], num);
            num = fma(-z2, o[plane], num);
            nw = fma(zh[q], num, A.om1 * old);
          }
          Ec[off] = nw;
          if (A.check == 0) {
            const u64 b = (u64)__double_as_longlong(fabs(nw - old));
            big = b > big ? b : big;
          }
        }
        const int ye = jj == 0 && s.jb > 0 ? edge_ylo(kk) : jj == s.nyb - 1 && s.jb + 1 < A.gy ? edge_yhi(A.bz, kk) : -1;
        const int ze = kk == 0 && s.kb > 0 ? edge_zlo(A.bz, jj)
                       : kk == s.nzb - 1 && s.kb + 1 < A.gz ? edge_zhi(A.by, A.bz, jj) : -1;
        if (ye >= 0 || ze >= 0) {
          const u64 v = (u64)__double_as_longlong(nw);
          const u64 lo = tagged((unsigned)v, seq), hi = tagged((unsigned)(v >> 32), seq);
          if (ye >= 0) st_pair(mine + c * cstride + (ye * nh + m) * 2, lo, hi);
          if (ze >= 0) st_pair(mine + c * cstride + (ze * nh + m) * 2, lo, hi);
        }
      }
      if (c == 1 && A.check == 0) {
        big = warp_max_bits(big);
        if ((t & 31) == 0 && big != 0) atomicMax(A.errs + sweep, big);
        big = 0;
      }
      unsigned pend = 0;
#pragma unroll
      for (int n = 0; n < kHalo; ++n) pend |= hdst[n] >= 0 ? 1u << n : 0u;
      for (int it = 0; pend != 0; ++it) {
        u64 v[kHalo][2];
#pragma unroll
        for (int n = 0; n < kHalo; ++n)
          if (pend >> n & 1) ld_pair(hsrc[n] + c * cstride, v[n][0], v[n][1]);
#pragma unroll
        for (int n = 0; n < kHalo; ++n)
          if ((pend >> n & 1) && (unsigned)(v[n][0] >> 32) == seq + A.skew && (unsigned)(v[n][1] >> 32) == seq + A.skew) {
            Ec[hdst[n]] = __longlong_as_double((long long)((v[n][1] << 32) | (v[n][0] & 0xffffffffull)));
            pend &= ~(1u << n);
          }
        if (pend != 0 && (it & 255) == 255 && (it > A.polls || ld_flag(A.err) != 0)) {
          fail = true;
          break;
        }
      }
      if (__syncthreads_or(fail)) {
        if (t == 0) atomicExch(A.err, 1);
        return;
      }
    }
    if (A.check > 0 && (A.sweep0 + sweep + 1) % A.check == 0) {
      u64 res = 0;
      for (int it = t; it < items; it += nt) {
        const unsigned ps = pos[it];
        const int m = ps & 4095u, jj = ps >> 12 & 1023u, kk = ps >> 22 & 255u;
        const int off = (kk + 1) * plane + (jj + 1) * Ld + m + 1;
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if (ps >> (30 + c) & 1) {
            const double* o = E + (1 - c) * all + off;
            const bool first = (c == 0) == (((s.j0 + jj + s.k0 + kk) & 1) == 1);
            const int i = (first ? 2 : 3) + 2 * m;
            const double bd = B[c * allB + it], own = E[c * all + off];
            const double W = first ? o[-1] : o[0], Ea = first ? o[0] : o[1];
            const double a0 = X[i - 1], a2 = X[2 * (d.nx + 1) + i - 1];
            const double y0 = Y[jj], y2 = Y[2 * A.by + jj], z0 = Z[kk], z2 = Z[2 * A.bz + kk];
            double r;
            if (EXACT) {
              const double num = bd - a0 * W - a2 * Ea - y0 * o[-Ld] - y2 * o[Ld] - z0 * o[-plane] - z2 * o[plane];
              r = num - dg[c * allB + it] * own;
            } else {
              double q = a0 * W;
              q = fma(a2, Ea, q);
              q = fma(y0, o[-Ld], q);
              q = fma(y2, o[Ld], q);
              q = fma(z0, o[-plane], q);
              q = fma(z2, o[plane], q);
              q = fma(X[d.nx + 1 + i - 1] + Y[A.by + jj] + Z[A.bz + kk], own, q);
              r = bd - q;
            }
            const u64 b = (u64)__double_as_longlong(fabs(r));
            res = b > res ? b : res;
          }
      }
      res = warp_max_bits(res);
      if ((t & 31) == 0 && res != 0) atomicMax(A.errs + sweep, res);
      __syncthreads();   // the next red pass overwrites the values that the residual has read
    }
  }
  for (int it = t; it < items; it += nt) {
    const unsigned ps = pos[it];
    const int m = ps & 4095u, jj = ps >> 12 & 1023u, kk = ps >> 22 & 255u, j = s.j0 + jj, k = s.k0 + kk;
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (ps >> (30 + c) & 1) {
        const int i = ((c == 0) == (((j + k) & 1) == 1) ? 2 : 3) + 2 * m;
        A.pc_out[d.at(i, j, k)] = E[c * all + (kk + 1) * plane + (jj + 1) * Ld + m + 1];
      }
  }
}

// -------------------------------------------------------------------------- plans

namespace {

// The split of ny x nz rows over at most nsm blocks that ends a pass soonest: the
// shared-memory cycles of the busiest block's rows (0.75 a group), the march of its
// threads through zl planes (about 130 cycles each, one after the other) and its ghost
// rows. Every block has at least two rows each way, so that no row is both edges, and
// its row positions have a thread each.
void split_rows32(int nq, int ny, int nz, int nsm, ResidentPlan& pl) {
  double best = 1e300;
  for (int gy = 1; gy <= std::min(ny / 2, nsm); ++gy)
    for (int gz = 1; gz <= std::min(nz / 2, nsm / gy); ++gz) {
      const int by = (ny + gy - 1) / gy, bz = (nz + gz - 1) / gz, cols = by * nq;
      if (cols > kMaxThreads) continue;
      const int chunks = std::min(kMaxThreads / cols, bz), zl = (bz + chunks - 1) / chunks;
      const int ghosts = 2 * ((gy > 1 ? bz : 0) + (gz > 1 ? by : 0)) * nq;
      const double cost = std::max(0.75 * by * bz * nq, 130.0 * zl) + 0.3 * ghosts;
      if (cost < best && 2 * (by + bz) * nq <= kHalo * kMaxThreads) {
        best = cost;
        pl.gy = gy; pl.gz = gz; pl.by = by; pl.bz = bz; pl.zl = zl;
        const int owners = cols * ((bz + zl - 1) / zl);
        pl.nt = std::min(kMaxThreads, (owners + ghosts + 31) / 32 * 32);
        while (kHalo * pl.nt < 2 * (by + bz) * nq) pl.nt += 32;
      }
    }
}

}  // namespace

ResidentPlan plan_resident32(int nx, int ny, int nz, int nsm) {
  ResidentPlan pl;
  const int nq = row_groups(nx);
  split_rows32(nq, ny, nz, nsm, pl);
  if (pl.gy == 0) return pl;
  const size_t all = (size_t)(pl.bz + 2) * (pl.by + 2) * (4 * nq + 8), rows = (size_t)pl.by * pl.bz * 4 * nq;
  pl.smem = (2 * all + 2 * rows + 4 * (size_t)pl.bz) * sizeof(float);
  pl.xch_words = (size_t)pl.gy * pl.gz * 2 * 2 * (pl.by + pl.bz) * 4 * nq;
  pl.ok = pl.smem <= kSmemCap;
  return pl;
}

namespace {
template <int NH>
cudaError_t go32(const ResidentPlan& pl, Resident32& a, cudaStream_t st) {
  const void* k = (const void*)k_resident32<NH>;
  const cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(k, dim3((unsigned)(pl.gy * pl.gz)), dim3((unsigned)pl.nt), args, pl.smem, st);
}
}  // namespace

cudaError_t launch_resident32(const ResidentPlan& pl, Resident32 a, cudaStream_t st) {
  a.gy = pl.gy; a.gz = pl.gz; a.by = pl.by; a.bz = pl.bz; a.zl = pl.zl;
  const int nh = (2 * (pl.by + pl.bz) * row_groups(a.d.nx) + pl.nt - 1) / pl.nt;
  return nh <= 1 ? go32<1>(pl, a, st) : nh <= 2 ? go32<2>(pl, a, st) : go32<kHalo>(pl, a, st);
}

// The split for the FP64 form: bound by the FP64 pipe, so the busiest block's rows count
// first, then its edge rows.
ResidentPlan plan_resident64(int nx, int ny, int nz, int nsm, bool exact) {
  ResidentPlan pl;
  const int nh = (nx + 1) >> 1;
  double best = 1e300;
  for (int gy = 1; gy <= std::min(ny / 2, nsm); ++gy)
    for (int gz = 1; gz <= std::min(nz / 2, nsm / gy); ++gz) {
      const int by = (ny + gy - 1) / gy, bz = (nz + gz - 1) / gz;
      const double cost = (double)by * bz + 0.15 * ((gy > 1 ? 2 * bz : 0) + (gz > 1 ? 2 * by : 0));
      if (cost < best) {
        best = cost;
        pl.gy = gy; pl.gz = gz; pl.by = by; pl.bz = bz;
      }
    }
  if (pl.gy == 0 || nh > 4095 || pl.by > 1023 || pl.bz > 255) return pl;
  const int items = pl.by * pl.bz * nh, ghosts = 2 * (pl.by + pl.bz) * nh;
  pl.nt = std::min(kMaxThreads, (items + 31) / 32 * 32);
  while (pl.nt < kMaxThreads && kHalo * pl.nt < ghosts) pl.nt += 32;
  const size_t all = (size_t)(pl.bz + 2) * (pl.by + 2) * (nh + 2);
  pl.smem = (2 * all + (exact ? 8 : 4) * (size_t)items + 3 * (size_t)(nx + 1) + 3 * (size_t)(pl.by + pl.bz)) * sizeof(double) +
            (size_t)items * sizeof(unsigned);
  pl.xch_words = (size_t)pl.gy * pl.gz * 2 * 2 * (pl.by + pl.bz) * 2 * nh;
  pl.ok = kHalo * pl.nt >= ghosts && pl.smem <= kSmemCap;
  return pl;
}

cudaError_t launch_resident64(const ResidentPlan& pl, Resident64 a, bool exact, cudaStream_t st) {
  a.gy = pl.gy; a.gz = pl.gz; a.by = pl.by; a.bz = pl.bz;
  const void* k = exact ? (const void*)k_resident64<true> : (const void*)k_resident64<false>;
  const cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(k, dim3((unsigned)(pl.gy * pl.gz)), dim3((unsigned)pl.nt), args, pl.smem, st);
}

// The exchange buffer of a context, at least `words` long, zeroed when it is new (pass
// numbers start at 1). The forms share it, so the old one stays until there is a larger one.
static bool ensure_exchange(ib3d_ctx* c, size_t words) {
  if (words <= c->xch_words) return true;
  u64* p = nullptr;
  if (cudaMalloc(&p, words * sizeof(u64)) != cudaSuccess ||
      cudaMemsetAsync(p, 0, words * sizeof(u64), c->st) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(p);
    return false;
  }
  cudaStreamSynchronize(c->st);
  cudaFree(c->xch);
  c->xch = p;
  c->xch_words = words;
  c->xch_seq = 0;
  return true;
}

// The second array of the FP64 batches and their recorded measures: all of them, or none.
constexpr int kBatch = 256;   // sweeps of an FP64 batch, at most
static bool ensure_batches(ib3d_ctx* c) {
  if (c->pc2) return true;
  if (cudaMalloc(&c->pc2, (size_t)c->d.n3 * sizeof(double)) == cudaSuccess &&
      cudaMalloc(&c->d_errs, (kBatch + 1) * sizeof(u64)) == cudaSuccess &&
      cudaMallocHost(&c->h_errs, (kBatch + 1) * sizeof(u64)) == cudaSuccess)
    return true;
  cudaGetLastError();
  cudaFree(c->pc2);
  cudaFree(c->d_errs);
  c->pc2 = nullptr;
  c->d_errs = c->h_errs = nullptr;   // the last one of the three, so never there when one has failed
  return false;
}

// One pass of the defect correction on chip: n FP32 sweeps on the packed right-hand side
// from e = 0, then pc += e. False (and nothing done) where the grid does not fit, or the
// device cannot hold all blocks at once; the caller then launches the passes one by one.
bool run_resident32(ib3d_ctx* c, int n, int nsmooth, int nramp, double wi, float om, float om1) {
  if (!c->res32_planned) {
    c->res32_planned = true;
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
    if (coop && c->ep[0]) c->res32 = plan_resident32(c->d.nx, c->d.ny, c->d.nz, c->nsm);
    if (c->res32.ok && !ensure_exchange(c, c->res32.xch_words)) c->res32.ok = false;
  }
  if (!c->res32.ok) return false;
  Resident32 a{};
  a.d = c->d;
  for (int q = 0; q < 3; ++q) {
    a.axp[0][q] = c->g.axp[0][q];
    a.axp[1][q] = c->g.axp[1][q];
    a.ay[q] = c->g.acy32[q];
    a.az[q] = c->g.acz32[q];
  }
  const size_t first = ((size_t)c->d.NY2 + 1) * c->packed_lp + 4;   // row (2, 2), entry 0
  a.r[0] = c->rp[0] + first;
  a.r[1] = c->rp[1] + first;
  a.rs = c->packed_lp;
  a.ps = c->packed_lp * c->d.NY2;
  a.pc = c->pc;
  a.xch = c->xch;
  a.seq0 = c->xch_seq;
  a.nsweeps = n;
  a.nsmooth = nsmooth;
  a.nramp = nramp;
  a.wi = wi;
  a.om = om;
  a.om1 = om1;
  a.err = &c->ctl->stage_err;
  a.polls = c->polls;
  a.skew = c->poll_skew;
  if (launch_resident32(c->res32, a, c->st) != cudaSuccess) {
    cudaGetLastError();
    c->res32.ok = false;
    return false;
  }
  c->xch_seq += 2u * (unsigned)n;
  return true;
}

// Is the diagonal of every cell of one sign and of a size that div_known takes?
static bool plain_diagonal(const ib3d_ctx* c) {
  const int n[3] = {c->d.nx, c->d.ny, c->d.nz};
  double lo = 0.0, hi = 0.0;
  for (int ax = 0; ax < 3; ++ax) {
    double l = 1e300, h = 0.0;
    for (int i = 1; i <= n[ax]; ++i) {
      const double v = -c->hac[ax][1][i];
      if (!(v > 0.0)) return false;
      l = std::min(l, v);
      h = std::max(h, v);
    }
    lo += l;
    hi += h;
  }
  return lo > 0x1p-200 && hi < 0x1p200;
}

// A whole FP64 solve (REDBLACKSOR) in batches of on-chip sweeps: k_sor64's arithmetic, or
// k_sor64_fast's. Returns false (and nothing done) where the grid does not fit; rc is the
// solve's result otherwise. Each batch goes from one array to the other, so a batch in
// which the stopping test is met runs again from its input up to that sweep; the batches
// grow to 256 sweeps and shrink as the measured rate says that the end is near.
bool run_resident64(ib3d_ctx* c, ib3d_solve_stats* st, bool exact, int& rc) {
  ResidentPlan& pl = exact ? c->res64 : c->res64f;
  bool& planned = exact ? c->res64_planned : c->res64f_planned;
  if (!planned) {
    planned = true;
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
    if (coop) pl = plan_resident64(c->d.nx, c->d.ny, c->d.nz, c->nsm, exact);
    if (pl.ok && (!ensure_exchange(c, pl.xch_words) || !ensure_batches(c))) pl.ok = false;
  }
  if (!pl.ok || (exact && !plain_diagonal(c))) return false;
  const ib3d_params& P = c->prm;
  const size_t bytes = (size_t)c->d.n3 * sizeof(double);
  const bool resid = P.criterion == IB3D_CRIT_RESIDUAL;
  const int every = P.check_every < 1 ? 1 : P.check_every;
  Resident64 a{};
  a.d = c->d;
  for (int q = 0; q < 3; ++q) {
    a.ax[q] = c->g.acx[q];
    a.ay[q] = c->g.acy[q];
    a.az[q] = c->g.acz[q];
  }
  a.bdt = c->bdt;
  a.cell = c->cell;
  a.xch = c->xch;
  a.check = resid ? every : 0;
  a.omega = P.omega;
  a.om1 = 1.0 - P.omega;
  a.errs = c->d_errs;
  a.err = reinterpret_cast<int*>(c->d_errs + kBatch);
  a.polls = c->polls;
  a.skew = c->poll_skew;
  rc = IB3D_ERR_CUDA;
  auto failed = [&](const char* what) {
    c->err = what;
    rc = IB3D_ERR_CUDA;
    return true;
  };
  double *in = c->pc, *out = c->pc2;
  if (cudaMemcpyAsync(c->pc2, c->pc, bytes, cudaMemcpyDeviceToDevice, c->st) != cudaSuccess) return failed("FP64 sweeps: copy of pc");
  long long sweep = 0, launched = 0;
  int batch = 16, done = 0;
  double err = 0.0, last_res = 0.0, rate_err = 0.0;   // rate_err: the stopping measure at rate_at sweeps
  long long rate_at = 0;
  bool have_rate = false;
  while (!done) {
    PhaseScope ps(c, PH_SOR64);
    int n = (int)std::min<long long>(batch, P.max_sweeps - sweep);
    a.pc_in = in;
    a.pc_out = out;
    a.sweep0 = sweep;
    a.nsweeps = n;
    a.seq0 = c->xch_seq;
    if (cudaMemsetAsync(c->d_errs, 0, (kBatch + 1) * sizeof(u64), c->st) != cudaSuccess) return failed("FP64 sweeps: control words");
    const cudaError_t le = launch_resident64(pl, a, exact, c->st);
    if (le != cudaSuccess) {
      cudaGetLastError();
      pl.ok = false;
      if (launched == 0) return false;
      return failed("FP64 sweeps: cooperative launch refused");
    }
    ++launched;
    c->launches += 1;
    c->xch_seq += 2u * (unsigned)n;
    if (cudaMemcpyAsync(c->h_errs, c->d_errs, (kBatch + 1) * sizeof(u64), cudaMemcpyDeviceToHost, c->st) != cudaSuccess ||
        cudaStreamSynchronize(c->st) != cudaSuccess)
      return failed("FP64 sweeps: reading the convergence words");
    if ((int)c->h_errs[kBatch] != 0) return failed("FP64 sweeps: a neighbouring block's rows never arrived (bounded wait gave up)");
    int stop = 0;   // sweeps of this batch up to the decision
    for (int q = 1; q <= n && !done; ++q) {
      const long long at = sweep + q;
      const bool tested = !resid || at % every == 0;
      if (tested) {
        std::memcpy(&err, &c->h_errs[q - 1], sizeof(double));
        last_res = err;
        if (!(err >= P.eps)) done = 1;
      } else {
        err = last_res;
      }
      if (!done && at >= P.max_sweeps) done = 2;
      stop = q;
    }
    if (done == 1 && stop < n) {   // the test was met inside the batch: up to that sweep, from the same input
      a.nsweeps = stop;
      a.seq0 = c->xch_seq;
      if (launch_resident64(pl, a, exact, c->st) != cudaSuccess) return failed("FP64 sweeps: cooperative launch refused");
      c->launches += 1;
      c->xch_seq += 2u * (unsigned)stop;
      if (cudaMemcpyAsync(c->h_errs, c->d_errs, (kBatch + 1) * sizeof(u64), cudaMemcpyDeviceToHost, c->st) != cudaSuccess ||
          cudaStreamSynchronize(c->st) != cudaSuccess || (int)c->h_errs[kBatch] != 0)
        return failed("FP64 sweeps: a neighbouring block's rows never arrived (bounded wait gave up)");
    }
    sweep += stop;
    std::swap(in, out);
    batch = std::min(2 * batch, kBatch);
    if (!done && last_res > 0.0) {   // sweeps that the rate since the last batch still asks for
      if (have_rate && last_res < rate_err) {
        const double need = std::log(P.eps / last_res) / (std::log(last_res / rate_err) / (double)(sweep - rate_at));
        batch = std::max(16, (int)std::min((double)batch, 0.9 * need));
      }
      rate_err = last_res;
      rate_at = sweep;
      have_rate = true;
    }
  }
  if (in != c->pc && cudaMemcpyAsync(c->pc, in, bytes, cudaMemcpyDeviceToDevice, c->st) != cudaSuccess)
    return failed("FP64 sweeps: copy of pc");
  st->sweeps = sweep;
  st->outer = 0;
  c->t_sweeps64 += sweep;
  st->final_err = err;
  rc = err != err ? IB3D_ERR_NONFINITE : done == 2 ? IB3D_ERR_NOCONV : IB3D_OK;
  return true;
}

}  // namespace ib3d
