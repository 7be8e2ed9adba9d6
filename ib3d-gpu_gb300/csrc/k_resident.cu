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
// The blocks wait on one another, so the launch is cooperative (all blocks resident). A
// poll gives up after a bounded number of loads, or when another block has: the block then
// sets the error flag and every block returns without storing a result; nothing is in
// flight by then. The kernels run on one stream at a time per exchange buffer.
//
// Compiled with -fmad=false: the FP64 kernel keeps the reference's rounding.
#include <algorithm>

#include "resident.cuh"
#include "sor32_update.cuh"

namespace ib3d {

namespace {

typedef unsigned long long u64;

constexpr int kHalo = 4;                  // received items per thread, at most
constexpr int kPollLimit = 1 << 20;       // about half a second
constexpr int kMaxThreads = 512;
constexpr size_t kSmemCap = 227 * 1024 - 1024;

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
              if ((unsigned)(v[n][0] >> 32) == seq && (unsigned)(v[n][1] >> 32) == seq &&
                  (unsigned)(v[n][2] >> 32) == seq && (unsigned)(v[n][3] >> 32) == seq) {
                *reinterpret_cast<float4*>(E + c * all + hdst[n]) =
                    make_float4(__uint_as_float((unsigned)v[n][0]), __uint_as_float((unsigned)v[n][1]),
                                __uint_as_float((unsigned)v[n][2]), __uint_as_float((unsigned)v[n][3]));
                pend &= ~(1u << n);
              }
            }
          if (pend != 0 && (it & 255) == 255 && (it > kPollLimit || ld_flag(A.err) != 0)) {
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
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
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

// The exchange buffer of a context, at least `words` long, zeroed when it is new (pass
// numbers start at 1).
static bool ensure_exchange(ib3d_ctx* c, size_t words) {
  if (words <= c->xch_words) return true;
  cudaStreamSynchronize(c->st);
  cudaFree(c->xch);
  c->xch = nullptr;
  c->xch_words = 0;
  if (cudaMalloc(&c->xch, words * sizeof(u64)) != cudaSuccess ||
      cudaMemsetAsync(c->xch, 0, words * sizeof(u64), c->st) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(c->xch);
    c->xch = nullptr;
    return false;
  }
  c->xch_words = words;
  c->xch_seq = 0;
  return true;
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
  if (launch_resident32(c->res32, a, c->st) != cudaSuccess) {
    cudaGetLastError();
    c->res32.ok = false;
    return false;
  }
  c->xch_seq += 2u * (unsigned)n;
  return true;
}

}  // namespace ib3d
