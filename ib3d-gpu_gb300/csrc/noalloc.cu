// Pressure solve that allocates no memory.
//
// Some host codes that would call this library cannot call cudaMalloc: a Fortran
// or C++ solver whose device memory is owned by another runtime (an OpenACC data
// region, a framework's caching allocator, a fixed memory pool sized at start-up),
// a code that must not allocate inside its time loop for latency or fragmentation
// reasons, or one that runs where allocation is forbidden. They hold their arrays
// already and only need the solve. ib3d_pressure_solve_noalloc takes every input
// and output as a device pointer the caller owns, and keeps its own scratch (the
// FP32 right-hand side and correction of the inner sweeps, and the loop's control
// block) in one file-scope __device__ array that the library image carries, so the
// call performs no allocation of any kind.
//
// The solve is the library's mixed-precision pressure solve: FP64 defect
// correction around FP32 red-black sweeps, stopped at an FP64 residual L-inf
// tolerance, with the same arithmetic as ib3d_poisson_solver's IB3D_PREC_FP32DC mode.
// Grids that the on-chip sweeps take (k_resident.cu: all but those of very long rows) run
// each pass in one launch from FP32 tables of the caller's coefficients; before, every
// sweep was two launches that converted nine FP64 coefficients per cell: 14.4 us a sweep
// at 96x64x64 against 2.9.
#include <mutex>

#include "resident.cuh"

namespace ib3d {
namespace {

// Largest padded grid, (nx+2)*(ny+2)*(nz+2), the scratch can hold: 2^21 cells
// (for example 126^3), i.e. two FP32 arrays of 8 MiB each plus the control block.
constexpr long long kMaxCells = 1ll << 21;
constexpr size_t kArrayBytes = (size_t)kMaxCells * sizeof(float);
constexpr size_t kCtlOffset = 2 * kArrayBytes;
// FP32 coefficient tables of the on-chip form, behind the control block
constexpr size_t kTabOffset = kCtlOffset + 256;
constexpr size_t kTabBytes = 128 * 1024;
constexpr size_t kScratchBytes = kTabOffset + kTabBytes;

// The scratch itself. Every GPU that loads the library holds it until the process
// exits. In host code this name is only a host-side stand-in for the device
// object, so host code never passes it to a kernel: it passes the device address
// obtained once per device with cudaGetSymbolAddress (below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

std::mutex g_mu;
constexpr int kMaxDevices = 64;
unsigned char* g_addr[kMaxDevices] = {};

// Device address of the scratch on the current device, looked up on the first
// call made on that device and cached. A call that meets any CUDA error drops the
// cached address (forget_scratch_address), so the next call looks it up again.
cudaError_t scratch_on_current_device(unsigned char** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_addr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_addr[dev];
  return cudaSuccess;
}

void forget_scratch_address() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  std::lock_guard<std::mutex> lock(g_mu);
  g_addr[dev] = nullptr;
}

struct Coefs {  // the caller's (n,3) column-major Acx/Acy/Acz (device)
  const double *ax, *ay, *az;
  int nx, ny, nz;
  __device__ __forceinline__ double x(int c, int m) const { return ax[(m - 1) + nx * c]; }
  __device__ __forceinline__ double y(int c, int m) const { return ay[(m - 1) + ny * c]; }
  __device__ __forceinline__ double z(int c, int m) const { return az[(m - 1) + nz * c]; }
};

__device__ __forceinline__ void decide(SolveCtl* ctl, long long sweeps, double eps, long long max_sweeps) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned ticket = atomicAdd(&ctl->tickets, 1u);
    if (ticket == gridDim.x - 1) {
      __threadfence();
      const double err = bits_to_double(atomicExch(&ctl->res, 0ull));
      ctl->tickets = 0;
      ctl->last_res = err;
      if (!(err >= eps)) { ctl->done = 1; ctl->nsweeps = sweeps; ctl->final_err = err; }
      else if (sweeps >= max_sweeps) { ctl->done = 2; ctl->nsweeps = sweeps; ctl->final_err = err; }
      __threadfence();
    }
  }
}

// r = b/dt - A pc on fluid cells (FP64), its maximum, and r rounded to FP32: in the padded
// layout (r32, 0 off the fluid cells), or colour-packed without padding rows (rp: [2][nz][ny]
// rows of 4 row_groups(nx) entries, NaN off the fluid cells).
__global__ void k_na_residual(Dims d, Coefs A, const double* __restrict__ b, double deltat,
                              const double* __restrict__ pc, const unsigned char* __restrict__ cell,
                              float* __restrict__ r32, float* __restrict__ rp, SolveCtl* ctl, long long sweeps, double eps,
                              long long max_sweeps) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (tid < (unsigned)d.nx * (unsigned)d.ny * (unsigned)d.nz) {
    const int i = (int)(tid % (unsigned)d.nx) + 2;
    const unsigned t = tid / (unsigned)d.nx;
    const int j = (int)(t % (unsigned)d.ny) + 2, k = (int)(t / (unsigned)d.ny) + 2;
    const long long idx = d.at(i, j, k);
    float rr = rp ? __int_as_float(0x7fc00000) : 0.0f;
    if (cell[idx] == 0) {
      const long long sy = d.NX2, sz = (long long)d.NX2 * d.NY2;
      const double bdt = b[idx] / deltat;
      const double num = bdt - A.x(0, i - 1) * pc[idx - 1] - A.x(2, i - 1) * pc[idx + 1] -
                         A.y(0, j - 1) * pc[idx - sy] - A.y(2, j - 1) * pc[idx + sy] -
                         A.z(0, k - 1) * pc[idx - sz] - A.z(2, k - 1) * pc[idx + sz];
      const double diag = A.x(1, i - 1) + A.y(1, j - 1) + A.z(1, k - 1);
      const double r = num - diag * pc[idx];
      m = fabs(r);
      rr = (float)r;
    }
    if (rp) {
      const int L = 4 * row_groups(d.nx);
      const size_t half = (size_t)d.nz * d.ny * L;
      rp[(((i + j + k) & 1) ? 0 : half) + ((size_t)(k - 2) * d.ny + (j - 2)) * L + ((i - 2) >> 1)] = rr;
    } else {
      r32[idx] = rr;
    }
  }
  block_max_atomic(m, &ctl->res);
  decide(ctl, sweeps, eps, max_sweeps);
}

// The FP32 tables of the on-chip sweeps: the x coefficients grouped by four cells of one
// colour (Grid1D::axp: columns 1 and 3 negated, 0 beyond the row), then the y and the z
// columns, 1-based.
__global__ void k_na_tables(Coefs A, float* __restrict__ tab) {
  const int nq = row_groups(A.nx), nx4 = 24 * nq, ny3 = 3 * (A.ny + 1), nz3 = 3 * (A.nz + 1);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nx4 + ny3 + nz3; t += gridDim.x * blockDim.x) {
    float v = 0.f;
    if (t < nx4) {
      const int s = t / (12 * nq), c = (t / (4 * nq)) % 3, m = t % (4 * nq), i = 2 + s + 2 * m;
      if (i <= A.nx + 1) v = (float)A.x(c, i - 1) * (c == 1 ? 1.f : -1.f);
    } else if (t < nx4 + ny3) {
      const int c = (t - nx4) / (A.ny + 1), m = (t - nx4) % (A.ny + 1);
      if (m >= 1) v = (float)A.y(c, m);
    } else {
      const int c = (t - nx4 - ny3) / (A.nz + 1), m = (t - nx4 - ny3) % (A.nz + 1);
      if (m >= 1) v = (float)A.z(c, m);
    }
    tab[t] = v;
  }
}

// One colour of the FP32 red-black sweep on A e = r, in place.
template <int COLOR>
__global__ void k_na_sor32(Dims d, Coefs A, const float* __restrict__ r32, float* __restrict__ e,
                           const unsigned char* __restrict__ cell, float omega, float om1) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned npairs = (unsigned)(d.nx + 1) >> 1;
  if (tid >= npairs * (unsigned)d.ny * (unsigned)d.nz) return;
  const int ip = (int)(tid % npairs);
  const unsigned t = tid / npairs;
  const int j = (int)(t % (unsigned)d.ny) + 2, k = (int)(t / (unsigned)d.ny) + 2;
  const int i0 = 2 + 2 * ip;
  const int i = i0 + ((i0 + j + k + 1 + COLOR) & 1);
  if (i > d.nx + 1) return;
  const long long idx = d.at(i, j, k);
  if (cell[idx] != 0) return;
  const long long sy = d.NX2, sz = (long long)d.NX2 * d.NY2;
  float num = r32[idx];
  num = fmaf(-(float)A.x(0, i - 1), e[idx - 1], num);
  num = fmaf(-(float)A.x(2, i - 1), e[idx + 1], num);
  num = fmaf(-(float)A.y(0, j - 1), e[idx - sy], num);
  num = fmaf(-(float)A.y(2, j - 1), e[idx + sy], num);
  num = fmaf(-(float)A.z(0, k - 1), e[idx - sz], num);
  num = fmaf(-(float)A.z(2, k - 1), e[idx + sz], num);
  const float diag = (float)A.x(1, i - 1) + (float)A.y(1, j - 1) + (float)A.z(1, k - 1);
  e[idx] = sor32_update(e[idx], num, diag, omega, om1);
}

__global__ void k_na_accumulate(long long n3, double* __restrict__ pc, float* __restrict__ e) {
  const unsigned idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (unsigned)n3) return;
  const float x = e[idx];
  if (x != 0.0f) {
    pc[idx] = pc[idx] + (double)x;
    e[idx] = 0.0f;
  }
}

// The on-chip form's exchange buffer follows its right-hand side (two halves).
size_t exchange_offset(size_t half) { return (2 * half * sizeof(float) + 255) / 256 * 256; }

// The split of the on-chip sweeps where the grid, the exchange buffer and the tables fit.
bool plan_noalloc(int64_t nx, int64_t ny, int64_t nz, ResidentPlan& plan) {
  int dev = 0, nsm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return false;
  const size_t nq = (size_t)row_groups((int)nx);
  if ((24 * nq + 3 * (size_t)(ny + 1) + 3 * (size_t)(nz + 1)) * sizeof(float) > kTabBytes) return false;
  plan = plan_resident32((int)nx, (int)ny, (int)nz, nsm);
  return plan.ok && exchange_offset((size_t)ny * nz * 4 * nq) + plan.xch_words * 8 <= kCtlOffset;
}

constexpr int kNotResident = 1;   // the cooperative launch was refused before anything ran

// plan: the split of the on-chip sweeps, or null for one launch per colour pass.
int run_noalloc(const ResidentPlan* plan, int64_t nx, int64_t ny, int64_t nz, const double* acx, const double* acy, const double* acz,
                const unsigned char* cell, const double* b, double deltat, double* pc, double omega, double eps,
                int64_t max_sweeps, int32_t inner_sweeps, cudaStream_t st, unsigned char* base,
                int64_t* sweeps_out, double* residual_out) {
  const long long n3 = (nx + 2) * (ny + 2) * (nz + 2);
  float* r32 = reinterpret_cast<float*>(base);
  float* e32 = reinterpret_cast<float*>(base + kArrayBytes);
  SolveCtl* ctl = reinterpret_cast<SolveCtl*>(base + kCtlOffset);
  Dims d;
  d.nx = (int)nx; d.ny = (int)ny; d.nz = (int)nz;
  d.NX2 = d.nx + 2; d.NY2 = d.ny + 2; d.NZ2 = d.nz + 2;
  d.n3 = n3;
  const Coefs A{acx, acy, acz, d.nx, d.ny, d.nz};
  // the scratch keeps the previous call's contents: the correction must start at
  // zero and the control block must be cleared
  if (!plan && cudaMemsetAsync(e32, 0, (size_t)n3 * sizeof(float), st) != cudaSuccess) return IB3D_ERR_CUDA;
  if (cudaMemsetAsync(ctl, 0, sizeof(SolveCtl), st) != cudaSuccess) return IB3D_ERR_CUDA;
  Resident32 res{};
  if (plan) {
    const int nq = row_groups(d.nx);
    const size_t rows = (size_t)ny * nz, half = rows * 4 * nq;
    float* tab = reinterpret_cast<float*>(base + kTabOffset);
    for (int s = 0; s < 2; ++s)
      for (int c = 0; c < 3; ++c) res.axp[s][c] = reinterpret_cast<const float4*>(tab) + (3 * s + c) * nq;
    for (int c = 0; c < 3; ++c) {
      res.ay[c] = tab + 24 * nq + c * (ny + 1);
      res.az[c] = tab + 24 * nq + 3 * (ny + 1) + c * (nz + 1);
    }
    res.d = d;
    res.r[0] = r32;
    res.r[1] = r32 + half;
    res.rs = 4 * nq;
    res.ps = d.ny * 4 * nq;
    res.pc = pc;
    res.xch = reinterpret_cast<unsigned long long*>(base + exchange_offset(half));
    res.nsweeps = inner_sweeps;
    res.om = (float)omega;
    res.om1 = (float)(1.0 - omega);
    res.err = &ctl->stage_err;
    res.polls = kPollLimit;
    // the rows' entries past their last cell stay NaN; the pass numbers start over
    if (cudaMemsetAsync(r32, 0xff, 2 * half * sizeof(float), st) != cudaSuccess) return IB3D_ERR_CUDA;
    if (cudaMemsetAsync(res.xch, 0, plan->xch_words * 8, st) != cudaSuccess) return IB3D_ERR_CUDA;
    k_na_tables<<<16, kBlock, 0, st>>>(A, tab);
  }
  const long long ncell = (long long)nx * ny * nz;
  const unsigned gres = (unsigned)((ncell + kBlock - 1) / kBlock);
  const unsigned gcol = (unsigned)((((nx + 1) / 2) * ny * nz + kBlock - 1) / kBlock);
  const unsigned gall = (unsigned)((n3 + kBlock - 1) / kBlock);
  const float om = (float)omega, om1 = (float)(1.0 - omega);
  SolveCtl h{};
  long long sweeps = 0;
  for (;;) {
    k_na_residual<<<gres, kBlock, 0, st>>>(d, A, b, deltat, pc, cell, r32, plan ? r32 : nullptr, ctl, sweeps,
                                              eps, max_sweeps);
    if (cudaGetLastError() != cudaSuccess) return IB3D_ERR_CUDA;
    if (cudaMemcpyAsync(&h, ctl, sizeof(SolveCtl), cudaMemcpyDeviceToHost, st) != cudaSuccess) return IB3D_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return IB3D_ERR_CUDA;
    if (h.stage_err) return IB3D_ERR_CUDA;   // a bounded wait of the on-chip sweeps gave up
    if (h.done) break;
    if (plan) {
      if (launch_resident32(*plan, res, st) != cudaSuccess) {
        cudaGetLastError();
        return sweeps == 0 ? kNotResident : IB3D_ERR_CUDA;
      }
      res.seq0 += 2u * (unsigned)inner_sweeps;
      sweeps += inner_sweeps;
      continue;
    }
    for (int q = 0; q < inner_sweeps; ++q) {
      k_na_sor32<0><<<gcol, kBlock, 0, st>>>(d, A, r32, e32, cell, om, om1);
      k_na_sor32<1><<<gcol, kBlock, 0, st>>>(d, A, r32, e32, cell, om, om1);
    }
    k_na_accumulate<<<gall, kBlock, 0, st>>>(n3, pc, e32);
    sweeps += inner_sweeps;
  }
  if (sweeps_out) *sweeps_out = h.nsweeps;
  if (residual_out) *residual_out = h.final_err;
  if (h.final_err != h.final_err) return IB3D_ERR_NONFINITE;
  return h.done == 2 ? IB3D_ERR_NOCONV : IB3D_OK;
}
}  // namespace
}  // namespace ib3d

using namespace ib3d;

extern "C" int ib3d_pressure_solve_noalloc(int64_t nx, int64_t ny, int64_t nz, const double* acx, const double* acy,
                                           const double* acz, const unsigned char* cell, const double* b,
                                           double deltat, double* pc, double omega, double eps,
                                           int64_t max_sweeps, int32_t inner_sweeps, void* stream,
                                           int64_t* sweeps_out, double* residual_out) {
  if (nx < 4 || ny < 4 || nz < 4 || !acx || !acy || !acz || !cell || !b || !pc || !(deltat > 0) ||
      !(omega > 0 && omega < 2) || !(eps > 0) || max_sweeps < 1 || inner_sweeps < 1)
    return IB3D_ERR_ARG;
  // each extent is bounded before the product is formed, so the product cannot overflow
  if (nx > kMaxCells || ny > kMaxCells || nz > kMaxCells) return IB3D_ERR_TOO_LARGE;
  if ((nx + 2) * (ny + 2) > kMaxCells) return IB3D_ERR_TOO_LARGE;
  const long long n3 = (nx + 2) * (ny + 2) * (nz + 2);
  if (n3 > kMaxCells) return IB3D_ERR_TOO_LARGE;
  unsigned char* base = nullptr;
  if (scratch_on_current_device(&base) != cudaSuccess) {
    forget_scratch_address();
    return IB3D_ERR_CUDA;
  }
  ResidentPlan plan;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = kNotResident;
  if (plan_noalloc(nx, ny, nz, plan))
    rc = run_noalloc(&plan, nx, ny, nz, acx, acy, acz, cell, b, deltat, pc, omega, eps, max_sweeps, inner_sweeps, st,
                     base, sweeps_out, residual_out);
  if (rc == kNotResident)
    rc = run_noalloc(nullptr, nx, ny, nz, acx, acy, acz, cell, b, deltat, pc, omega, eps, max_sweeps, inner_sweeps, st,
                     base, sweeps_out, residual_out);
  if (rc == IB3D_ERR_CUDA) forget_scratch_address();
  return rc;
}
