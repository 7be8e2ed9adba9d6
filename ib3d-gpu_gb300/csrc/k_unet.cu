// Kernels of the learned warm start: a small 3-D U-Net in BF16 with FP32
// accumulation (forward, backward, Adam). Host orchestration is in unet.cu.
//
// Activations are channels-last BF16 tensors [voxel][channel] over B x D x H x W
// voxels; a tensor can be a channel slice of a wider buffer (channel stride cs,
// offset co), which is how the U-Net's skip concatenations are stored. Channel
// counts are multiples of 16.
//
// 3x3x3 convolutions (zero padding) are implicit GEMMs on the fifth-generation
// tensor cores (tcgen05.mma kind::f16, BF16 operands from shared memory, FP32
// accumulator in tensor memory): rows are voxels, columns the output channels, and the
// reduction runs over 27 taps x input channels in steps of 16 channels. The voxels are
// numbered along rows that end in one zero (struct Seq), so that a tap is a constant
// distance in that numbering, and a block keeps a run of it in shared memory once: eight
// channels of a voxel are 16 bytes, voxel after voxel, one such line per eight channels.
// That is the canonical no-swizzle layout in both directions -- K-major for the
// convolution, whose reduction runs over channels, and MN-major for the weight gradient,
// whose reduction runs over voxels -- so all 27 taps' operands are the same bytes at 27
// start addresses, and nothing is gathered, copied or transposed per tap. The same
// kernel computes the input gradient with mirrored taps and transposed weights.
#include <cuda_bf16.h>

#include <algorithm>

#include "ib3d_internal.cuh"
#include "unet.cuh"

namespace ib3d {
namespace unet {

namespace {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle, K-major: core matrices of 8 rows x 16
// bytes; lbo = byte distance between core matrices along K, sbo = along M/N.
__device__ __forceinline__ unsigned long long smem_desc(const void* p, unsigned lbo, unsigned sbo) {
  unsigned long long d = (unsigned long long)((smem_addr(p) & 0x3FFFF) >> 4);
  d |= (unsigned long long)((lbo >> 4) & 0x3FFF) << 16;
  d |= (unsigned long long)((sbo >> 4) & 0x3FFF) << 32;
  d |= 1ull << 46;   // descriptor version; base offset 0, no swizzle
  return d;
}

// Bounded wait on an mbarrier phase (true when it completed).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned phase, int limit) {
  for (int it = 0; it < limit; ++it) {
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(phase) : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void decode(long long m, const Vol& v, int& b, int& z, int& y, int& x) {
  x = (int)(m % v.W);
  long long t = m / v.W;
  y = (int)(t % v.H);
  t /= v.H;
  z = (int)(t % v.D);
  b = (int)(t / v.D);
}

}  // namespace

// The voxels in the order of the shared-memory runs: rows of Wp entries, the last of
// which (x = W) is a zero that serves as the right neighbour of its row and the left
// neighbour of the next; Hp = H + 1 rows a plane, the last one zeros for both planes it
// lies between. A tap (dy, dx) is then the distance dy Wp + dx. Rows wider than 128 are
// cut into strips of 64 with a voxel of the neighbouring strips (or a zero) at both ends.
struct Seq {
  int W, H, D, Ws, ns, hl, Wp, Hp;   // Ws voxels of a row in a strip, ns strips, hl: 1 with ends of their own
  long long n;                       // entries
};
inline Seq make_seq(const Vol& v) {
  Seq q;
  q.W = v.W; q.H = v.H; q.D = v.D;
  q.Hp = v.H + 1;
  if (v.W <= 128) {
    q.Ws = v.W; q.ns = 1; q.hl = 0; q.Wp = v.W + 1;
  } else {
    q.Ws = 64; q.ns = (v.W + 63) / 64; q.hl = 1; q.Wp = 66;
  }
  q.n = (long long)v.B * v.D * q.ns * q.Hp * q.Wp;
  return q;
}
// Entry q: its plane bz = b D + z, its y and x; in: it holds a voxel, out: a voxel of its own
// (not a neighbouring strip's).
struct Entry {
  int bz, y, x;
  bool in, out;
};
__device__ __forceinline__ Entry seq_entry(const Seq& s, long long q) {
  Entry e{0, 0, 0, false, false};
  if (q < 0 || q >= s.n) return e;
  const unsigned u = (unsigned)q;   // fewer than 2^31 entries (checked at launch)
  const unsigned r = u / (unsigned)s.Wp, xp = u - r * (unsigned)s.Wp;
  const unsigned p = r / (unsigned)s.Hp;
  e.y = (int)(r - p * (unsigned)s.Hp);
  e.bz = (int)(p / (unsigned)s.ns);
  e.x = (int)(p - (unsigned)e.bz * (unsigned)s.ns) * s.Ws + (int)xp - s.hl;
  e.in = e.x >= 0 && e.x < s.W && e.y < s.H;
  e.out = e.in && (s.hl == 0 || (xp >= 1u && xp <= (unsigned)s.Ws));
  return e;
}

// 16 bytes to shared memory, or zeros.
__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_addr(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" :: "n"(PENDING) : "memory");
}

// A descriptor moved on by `units` of 16 bytes: the start address is the low 14 bits, and
// the buffers lie below 2^18 bytes, so the sum stays inside them. One thread issues the MMAs
// of an accumulator, so what it computes per MMA is time the tensor core waits: building a
// descriptor for each took 158 cycles an MMA.
__device__ __forceinline__ unsigned long long desc_at(unsigned long long d, int units) {
  return d + (unsigned long long)(long long)units;
}

__device__ __forceinline__ void mma_f16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool add) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
               " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u) : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned addr, unsigned (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__host__ __device__ constexpr unsigned tmem_cols(int n) { return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : n <= 256 ? 256u : 512u; }

// The runs of entries [q0, q0 + len) of nz planes at distances dz0, dz0 + step, ..., K
// channels: K / 8 lines of len 16-byte entries each, from dst.
__device__ __forceinline__ void load_runs(const Seq& s, const Act& X, int K, long long q0, int len, int dz0, int step,
                                          int nz, char* dst) {
  for (int i = threadIdx.x; i < len * nz; i += blockDim.x) {   // an entry of a plane per thread
    const int n = (i >= len) + (i >= 2 * len), p = i - n * len, dz = dz0 + n * step;   // nz is at most 3
    const Entry e = seq_entry(s, q0 + p);
    const int z = e.bz % s.D + dz;
    const bool ok = e.in && z >= 0 && z < s.D;
    const bf16* src = ok ? X.p + (((long long)(e.bz + dz) * s.H + e.y) * s.W + e.x) * X.cs + X.co : X.p;
    char* to = dst + ((size_t)n * (K >> 3) * len + p) * 16;
#pragma unroll 2
    for (int c = 0; c < K; c += 8, to += (size_t)len * 16) cp16(to, src + (ok ? c : 0), ok);
  }
}

// Y[v][n] = act( sum_{tap,k} X[v + sign*off(tap)][k] * Wt[n][tap][k] + bias[n] ),
// N output channels (a multiple of 16, at most 96). A block owns 128 R entries: R
// accumulators of 128 lanes x N FP32 columns in tensor memory. The three planes of the
// run and the weights of three taps at a time (a row dy of the stencil) pass through rings
// of NX and NB buffers, filled by asynchronous copies while one thread per accumulator
// issues the MMAs of what has arrived: nine steps of 3 taps x K / 16 MMAs per accumulator, in the order of
// the taps and channels, so that every output keeps one order of accumulation.
//
// Bound: a 128 x 16 operand is 4 KB of shared memory, 32 cycles, whatever N; at 8 x 32^3
// voxels and 16 channels 6 us of tensor time; measured 20 us against 62 us for a kernel
// that gathered every tap's operand through registers.
//
// Every wait is bounded and decided for the whole block: a barrier that does not
// complete sets *err, and the kernel still waits (bounded) for its issued MMAs
// before it frees the tensor memory.
constexpr int kConvThreads = 256;

template <int N>
__global__ void __launch_bounds__(kConvThreads) k_conv3(Seq seq, Act X, int K, const bf16* __restrict__ Wt,
                                                        const float* __restrict__ bias, int relu, int sign, Act Y, int R,
                                                        int NX, int NB, int* err) {
  static_assert(N % 16 == 0 && N >= 16 && N <= 96, "tcgen05 N");
  extern __shared__ __align__(128) char smc[];
  __shared__ __align__(8) unsigned long long bar[10];   // [0..8] steps, [9] all
  __shared__ unsigned tmem_base;
  const int t = threadIdx.x, warp = t >> 5;
  const int halo = seq.Wp + 1, len = 128 * R + 2 * halo;
  const size_t run = (size_t)len * K * 2, wstep = (size_t)3 * K * N * 2;   // bytes of a plane's run, of a step's weights
  char* sB = smc + NX * run;
  const unsigned cols = tmem_cols(R * N);
  const long long q0 = (long long)blockIdx.x * 128 * R;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmem_base)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 0) {
    for (int q = 0; q < 10; ++q)   // one arrival per accumulator's thread
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(&bar[q])), "r"(R));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base;
  // instruction descriptor: D FP32, A and B BF16, both K-major, N, M = 128
  const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) | ((128u >> 4) << 24);
  const int kch = K / 16;
  // of the first run's first line, and of the first weights
  const unsigned long long xdesc = smem_desc(smc, (unsigned)len * 16, 128), wdesc = smem_desc(sB, 128, 256);
  auto load_weights = [&](int g, char* dst) {
    const int chunks = 3 * N * (K / 8);
    for (int c = t; c < chunks; c += kConvThreads) {     // 8 input channels of output channel n, tap 3g + a
      const int o = c % (K / 8), r = c / (K / 8), n = r % N, a = r / N;
      cp16(dst + ((size_t)(a * kch + (o >> 1)) * N * 32 + (size_t)((n >> 3) * 2 + (o & 1)) * 128 + (n & 7) * 16),
           Wt + ((size_t)n * 27 + 3 * g + a) * K + 8 * o, true);
    }
  };
  const bool issuer = warp < R && (t & 31) == 0;   // warp m issues accumulator m's MMAs
  auto issue = [&](int g) {
    const unsigned long long ad0 = desc_at(xdesc, (g / 3 % NX) * (int)(run >> 4) + 128 * warp + halo +
                                                      sign * (g % 3 - 1) * seq.Wp);
    const unsigned long long bd0 = desc_at(wdesc, (g % NB) * (int)(wstep >> 4));
    const unsigned d = tmem + (unsigned)(warp * N);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      unsigned long long ad = desc_at(ad0, sign * (a - 1));
      unsigned long long bd = desc_at(bd0, a * kch * 2 * N);
#pragma unroll 2
      for (int kc = 0; kc < kch; ++kc) {
        mma_f16(d, ad, bd, idesc, g + a + kc > 0);
        ad = desc_at(ad, 2 * len);
        bd = desc_at(bd, 2 * N);
      }
    }
  };
  bool ok = true;
  if (NX == 3 && NB == 9) {   // everything fits: one load, one wait
    load_runs(seq, X, K, q0 - halo, len, -sign, sign, 3, smc);
    for (int g = 0; g < 9; ++g) load_weights(g, sB + g * wstep);
    cp_commit();
    cp_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // make it visible to the tensor core
    __syncthreads();
    if (issuer) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int g = 0; g < 9; ++g) issue(g);
      for (int g = 0; g < 9; ++g) mma_commit(&bar[g]);
    }
  } else {
    // step g = 3 (dz + 1) + dy + 1: taps 3g .. 3g + 2; the first step of a plane brings its run
    auto load_step = [&](int g) {
      if (g % 3 == 0) load_runs(seq, X, K, q0 - halo, len, sign * (g / 3 - 1), 0, 1, smc + (g / 3 % NX) * run);
      load_weights(g, sB + (g % NB) * wstep);
      cp_commit();
    };
    // a buffer of step g is free when the MMAs of the last step that read it are done
    auto last_reader = [&](int g) { return max(g - NB, g % 3 == 0 ? 3 * (g / 3 - NX) + 2 : -1); };
    int issued = 0;
    for (; issued < 9 && last_reader(issued) < 0; ++issued) load_step(issued);
    for (int g = 0; g < 9 && ok; ++g) {
      // step g has landed when at most issued - 1 - g later groups are pending
      switch (issued - 1 - g) {
        case 0: cp_wait<0>(); break;
        case 1: cp_wait<1>(); break;
        case 2: cp_wait<2>(); break;
        case 3: cp_wait<3>(); break;
        case 4: cp_wait<4>(); break;
        case 5: cp_wait<5>(); break;
        case 6: cp_wait<6>(); break;
        case 7: cp_wait<7>(); break;
        default: cp_wait<8>(); break;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (issuer) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue(g);
        mma_commit(&bar[g]);
      }
      // refill the buffers that earlier steps have read, and the next step's in any case
      while (issued < 9 && (last_reader(issued) < g || issued == g + 1) && ok) {
        ok = __syncthreads_and(mbar_wait(&bar[last_reader(issued)], 0, 1 << 20)) != 0;
        if (ok) load_step(issued++);
      }
    }
  }
  if (issuer) mma_commit(&bar[9]);   // arrives once every MMA of this thread is done
  bool done = __syncthreads_and(mbar_wait(&bar[9], 0, 1 << 20)) != 0;
  if (ok && done)   // the steps' own arrivals, so that none is left pending at exit
    for (int g = 0; g < 9; ++g) done = __syncthreads_and(mbar_wait(&bar[g], 0, 1 << 20)) != 0 && done;
  if (!ok || !done) {
    cp_wait<0>();                    // no copy is left in flight
    if (t == 0) atomicExch(err, 1);
    mbar_wait(&bar[9], 0, 1 << 20);  // let the issued MMAs finish before freeing the columns
  } else {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp < 4)
      for (int m = 0; m < R; ++m) {
        const Entry e = seq_entry(seq, q0 + 128 * m + t);
        const long long v = ((long long)e.bz * seq.H + e.y) * seq.W + e.x;
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
          unsigned r[16];
          tmem_ld16(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(m * N + c0), r);   // this warp's 32 lanes
          if (e.out) {
            bf16* dst = Y.p + v * Y.cs + Y.co + c0;
            __nv_bfloat162 h[8];
#pragma unroll
            for (int q = 0; q < 16; q += 2) {
              float v0 = __uint_as_float(r[q]), v1 = __uint_as_float(r[q + 1]);
              if (bias) { v0 += bias[c0 + q]; v1 += bias[c0 + q + 1]; }
              if (relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
              h[q >> 1] = __floats2bfloat162_rn(v0, v1);
            }
            reinterpret_cast<uint4*>(dst)[0] = *reinterpret_cast<const uint4*>(&h[0]);
            reinterpret_cast<uint4*>(dst)[1] = *reinterpret_cast<const uint4*>(&h[4]);
          }
        }
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(cols));
}

// dW[n][tap][k] += sum_v dZ[v][n] * X[v + off(tap)][k] on the tensor cores, the reduction
// over the entries of the sequence in steps of 16. Both operands are channels-last, so they
// are MN-major in the runs' layout; a tap is a start address in the X runs, and the
// gradient's run (zero where an entry is no voxel of its own) is the same for all. The runs of
// nz planes lie one behind the other, so their lines are evenly spaced, and one MMA covers
// the nz taps (dz, dy, dx) of a pair (dy, dx): D[n][dz][k], 64 lanes by nz K columns of
// tensor memory. A block has as many pairs as 512 columns hold and every gridDim.y-th chunk of
// 128 entries, two or more chunks in flight; at the end it stores its sums, and k_wgrad_sum adds
// those of all blocks in a fixed order (FP32 atomics on dW took 40 of 77 us).
//
// Bound: the gradient's 64 x 16 operand is 2 KB of shared memory, 16 cycles, per MMA, and the
// X operand nz K / 4: 14 us at 8 x 32^3 voxels and 16 x 16 channels. Measured there: 418 us
// for a kernel that gathered and transposed each tap's operand in registers, 100 with an
// MMA per tap and atomics, 58 now (the loads of one block per SM).
constexpr int kMaxStagesW = 4;
constexpr int kIssuersW = 4, kPairsPerIssuer = 3;   // 9 pairs at most

__global__ void __launch_bounds__(kConvThreads) k_wgrad_tc(Seq seq, Act dZ, int N, Act X, int K, float* __restrict__ part,
                                                           int nz, int pairs, int stages, int* err) {
  extern __shared__ __align__(128) char smc[];
  __shared__ __align__(8) unsigned long long bar[kMaxStagesW + 1];
  __shared__ unsigned tmem_base;
  const int t = threadIdx.x, warp = t >> 5;
  const int halo = seq.Wp + 1, len = 128 + 2 * halo;
  const int groups = (9 + pairs - 1) / pairs;                   // of pairs; blockIdx.x: planes, then groups
  const int zs = (int)blockIdx.x / groups, p0 = ((int)blockIdx.x % groups) * pairs, p1 = min(9, p0 + pairs);
  const size_t run = (size_t)len * K * 2, stage = nz * run + 8 * 128 * 16;   // the gradient's eight lines last
  const int chunks = (int)((seq.n + 127) / 128);
  const int mine = chunks > (int)blockIdx.y ? (chunks - 1 - (int)blockIdx.y) / (int)gridDim.y + 1 : 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmem_base)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 0) {
    for (int q = 0; q <= kMaxStagesW; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(&bar[q])), "r"(kIssuersW));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base;
  // instruction descriptor: D FP32, A and B BF16, both MN-major, N = nz K, M = 64
  const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((unsigned)(nz * K >> 3) << 17) |
                         ((64u >> 4) << 24);
  // warps 0 .. 3 issue the pairs p0 + warp, + 4, ...: distance of each pair's operand from the runs' start
  const bool issuer = warp < kIssuersW && (t & 31) == 0;
  int off[kPairsPerIssuer], npairs = 0;
#pragma unroll
  for (int u = 0; u < kPairsPerIssuer; ++u) {
    const int p = p0 + warp + kIssuersW * u;
    off[u] = halo + (p / 3 - 1) * seq.Wp + p % 3 - 1;
    npairs += p < p1;
  }
  const unsigned long long gdesc = smem_desc(smc + nz * run, 128, 128 * 16), xdesc = smem_desc(smc, 128, (unsigned)len * 16);
  auto load_chunk = [&](int i) {
    const long long q0 = ((long long)blockIdx.y + (long long)i * gridDim.y) * 128;
    char* s = smc + (i % stages) * stage;
    load_runs(seq, X, K, q0 - halo, len, zs - 1, 1, nz, s);
    char* g = s + nz * run;
    for (int p = t; p < 128; p += kConvThreads) {
      const Entry e = seq_entry(seq, q0 + p);
      const bf16* src = e.out ? dZ.p + (((long long)e.bz * seq.H + e.y) * seq.W + e.x) * dZ.cs + dZ.co : dZ.p;
      for (int c = 0; c < N; c += 8) cp16(g + ((size_t)(c >> 3) * 128 + p) * 16, src + (e.out ? c : 0), e.out);
    }
    cp_commit();
  };
  unsigned phase = 0;   // bit s: parity of stage s's next completion
  bool ok = true;
  for (int i = 0; i < stages - 1; ++i) {
    if (i < mine) load_chunk(i);
    else cp_commit();
  }
  for (int i = 0; i < mine && ok; ++i) {
    // chunk i has landed when only the stages - 2 chunks after it are pending
    if (stages == 2) cp_wait<0>();
    else if (stages == 3) cp_wait<1>();
    else cp_wait<2>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (issuer) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int at = (i % stages) * (int)(stage >> 4);
      unsigned long long ad = desc_at(gdesc, at), bd = desc_at(xdesc, at);
      for (int k = 0; k < 8; ++k) {
#pragma unroll
        for (int u = 0; u < kPairsPerIssuer; ++u)
          if (u < npairs) mma_f16(tmem + (unsigned)((warp + kIssuersW * u) * nz * K), ad, desc_at(bd, off[u]), idesc, i + k > 0);
        ad = desc_at(ad, 16);
        bd = desc_at(bd, 16);
      }
      mma_commit(&bar[i % stages]);
    }
    // while these run, chunk i + stages - 1 goes where chunk i - 1 was
    if (i >= 1) {
      const int sb = (i - 1) % stages;
      ok = __syncthreads_and(mbar_wait(&bar[sb], phase >> sb & 1u, 1 << 20)) != 0;
      phase ^= 1u << sb;
      if (!ok) break;
    }
    if (i + stages - 1 < mine) load_chunk(i + stages - 1);
    else cp_commit();
  }
  if (issuer) mma_commit(&bar[kMaxStagesW]);
  bool done = __syncthreads_and(mbar_wait(&bar[kMaxStagesW], 0, 1 << 20)) != 0;
  if (ok && done && mine > 0) {   // the last chunk's own arrival, so that none is left pending at exit
    const int sb = (mine - 1) % stages;
    done = __syncthreads_and(mbar_wait(&bar[sb], phase >> sb & 1u, 1 << 20)) != 0;
  }
  cp_wait<0>();
  if (!ok || !done) {
    if (t == 0) atomicExch(err, 1);
    mbar_wait(&bar[kMaxStagesW], 0, 1 << 20);   // let the issued MMAs finish before freeing the columns
  } else {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // rows 16 w .. 16 w + 15 of a 64-row accumulator lie in the first 16 lanes of warps w and
    // w + 4, which share the columns
    const int w4 = warp & 3, n = 16 * w4 + (t & 31);
    float* own = part + (size_t)blockIdx.y * N * 27 * K;
    if (16 * w4 < N)
      for (int q = warp >> 2; q < (p1 - p0) * nz * K / 16; q += 2) {
        const int p = p0 + q / (nz * K / 16), c0 = q % (nz * K / 16) * 16;
        unsigned r[16];
        tmem_ld16(tmem + ((unsigned)(w4 * 32) << 16) + (unsigned)(16 * q), r);
        if ((t & 31) < 16) {
          float4* to = reinterpret_cast<float4*>(own + ((size_t)n * 27 + 9 * (zs + c0 / K) + p) * K + c0 % K);
#pragma unroll
          for (int c = 0; c < 4; ++c)   // a block without chunks has no sums
            to[c] = mine > 0 ? make_float4(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1]),
                                           __uint_as_float(r[4 * c + 2]), __uint_as_float(r[4 * c + 3]))
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u));
}

// dW += the blocks' sums: eight threads of a column add every eighth block, then their sums
// in order. n: floats of a block's sums, a multiple of 4.
__global__ void __launch_bounds__(256) k_wgrad_sum(const float* __restrict__ part, int n, int blocks, float* __restrict__ dW) {
  __shared__ float4 sm[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = (blockIdx.x * 32 + lane) * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (e < n)
#pragma unroll 8
    for (int b = w; b < blocks; b += 8) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(part + (size_t)b * n + e));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < n) {
    for (int q = 1; q < 8; ++q) {
      const float4 v = sm[q][lane];
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const float4 v = *reinterpret_cast<const float4*>(dW + e);
    *reinterpret_cast<float4*>(dW + e) = make_float4(v.x + s.x, v.y + s.y, v.z + s.z, v.w + s.w);
  }
}

// dW[n][tap][k] += sum_v dZ[v][n] * X[v + off(tap)][k]   (FP32, CUDA cores): the
// reference form of k_wgrad_tc, kept for the gradient check of the tensor-core form.
// grid: (voxel chunks, 27 taps); each block reduces kWgTile voxels at a time through
// shared memory and adds its partial sums to dW with atomics.
constexpr int kWgTile = 32;
__global__ void __launch_bounds__(256) k_wgrad(Vol vol, Act dZ, int N, Act X, int K, float* __restrict__ dW,
                                               long long chunk) {
  extern __shared__ float sm[];
  float* sZ = sm;                    // [kWgTile][N]
  float* sX = sm + kWgTile * N;      // [kWgTile][K]
  const int tap = blockIdx.y;
  const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
  const long long M = vol.voxels();
  const long long v0 = (long long)blockIdx.x * chunk, v1 = min(M, v0 + chunk);
  const int NK = N * K;
  float acc[24];
#pragma unroll
  for (int q = 0; q < 24; ++q) acc[q] = 0.f;
  for (long long vt = v0; vt < v1; vt += kWgTile) {
    for (int e = threadIdx.x; e < kWgTile * N; e += blockDim.x) {
      const int lv = e / N, n = e % N;
      const long long m = vt + lv;
      sZ[e] = m < v1 ? __bfloat162float(dZ.p[m * dZ.cs + dZ.co + n]) : 0.f;
    }
    for (int e = threadIdx.x; e < kWgTile * K; e += blockDim.x) {
      const int lv = e / K, k = e % K;
      const long long m = vt + lv;
      float val = 0.f;
      if (m < v1) {
        int b, z, y, x;
        decode(m, vol, b, z, y, x);
        z += dz; y += dy; x += dx;
        if (z >= 0 && z < vol.D && y >= 0 && y < vol.H && x >= 0 && x < vol.W) {
          const long long sv = (((long long)b * vol.D + z) * vol.H + y) * vol.W + x;
          val = __bfloat162float(X.p[sv * X.cs + X.co + k]);
        }
      }
      sX[e] = val;
    }
    __syncthreads();
    for (int q = 0; q < 24; ++q) {
      const int pidx = threadIdx.x + q * 256;
      if (pidx >= NK) break;
      const int n = pidx / K, k = pidx % K;
      float s = acc[q];
#pragma unroll 8
      for (int lv = 0; lv < kWgTile; ++lv) s = fmaf(sZ[lv * N + n], sX[lv * K + k], s);
      acc[q] = s;
    }
    __syncthreads();
  }
  for (int q = 0; q < 24; ++q) {
    const int pidx = threadIdx.x + q * 256;
    if (pidx >= NK) break;
    const int n = pidx / K, k = pidx % K;
    atomicAdd(&dW[((size_t)n * 27 + tap) * K + k], acc[q]);
  }
}

// The elementwise kernels below move eight channels (16 bytes) per thread; channel counts,
// strides and offsets are multiples of 8.
struct Oct {
  __nv_bfloat162 h[4];
};
__device__ __forceinline__ Oct ld_oct(const bf16* p) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  return *reinterpret_cast<const Oct*>(&v);
}
__device__ __forceinline__ void st_oct(bf16* p, const Oct& o) { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&o); }
__device__ __forceinline__ void add_oct(float (&s)[8], const Oct& o) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 f = __bfloat1622float2(o.h[q]);
    s[2 * q] += f.x;
    s[2 * q + 1] += f.y;
  }
}

// ReLU backward through the layer's own output, in place, and the bias gradient:
// dY *= (Y > 0); db[n] += sum_v dY[v][n]. N is 16, 32 or 64, so a thread keeps its eight
// channels through the grid's strides, and a lane's sums combine with those of the lanes
// N / 8 apart. (Two kernels of one channel per thread took 29 us at 262,144 x 16.)
__global__ void __launch_bounds__(256) k_relu_bias_bwd(long long M, int N, Act dY, Act Y, float* __restrict__ db) {
  __shared__ float s[64];
  if (threadIdx.x < 64) s[threadIdx.x] = 0.f;
  __syncthreads();
  const int no = N >> 3, o = threadIdx.x % no;
  float a[8] = {};
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < M * no; e += (long long)gridDim.x * 256) {
    const long long m = e / no;
    bf16* p = dY.p + m * dY.cs + dY.co + 8 * o;
    const Oct y = ld_oct(Y.p + m * Y.cs + Y.co + 8 * o);
    Oct g = ld_oct(p);
    bool changed = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = __bfloat1622float2(y.h[q]);
      if (!(f.x > 0.f)) { g.h[q].x = __float2bfloat16(0.f); changed = true; }
      if (!(f.y > 0.f)) { g.h[q].y = __float2bfloat16(0.f); changed = true; }
    }
    if (changed) st_oct(p, g);
    add_oct(a, g);
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    for (int d = 16; d >= no; d >>= 1) a[q] += __shfl_xor_sync(0xffffffffu, a[q], d);
    if ((int)(threadIdx.x & 31) < no) atomicAdd(&s[8 * o + q], a[q]);
  }
  __syncthreads();
  if ((int)threadIdx.x < N) atomicAdd(&db[threadIdx.x], s[threadIdx.x]);
}

// 2x2x2 average pooling: out has half the extent of in along each axis.
__global__ void k_pool_fwd(Vol out, int C, Act in, Act o) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int no = C >> 3;
  if (e >= out.voxels() * no) return;
  const long long m = e / no;
  const int c = 8 * (int)(e - m * no);
  int b, z, y, x;
  decode(m, out, b, z, y, x);
  const int D2 = out.D * 2, H2 = out.H * 2, W2 = out.W * 2;
  float s[8] = {};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long sv = (((long long)b * D2 + 2 * z + (q >> 2)) * H2 + 2 * y + ((q >> 1) & 1)) * W2 + 2 * x + (q & 1);
    add_oct(s, ld_oct(in.p + sv * in.cs + in.co + c));
  }
  Oct r;
#pragma unroll
  for (int q = 0; q < 4; ++q) r.h[q] = __floats2bfloat162_rn(0.125f * s[2 * q], 0.125f * s[2 * q + 1]);
  st_oct(o.p + m * o.cs + o.co + c, r);
}

// gin[child] (+)= gout[parent] / 8
__global__ void k_pool_bwd(Vol out, int C, Act gout, Act gin, int accumulate) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int no = C >> 3;
  if (e >= out.voxels() * no) return;
  const long long m = e / no;
  const int c = 8 * (int)(e - m * no);
  int b, z, y, x;
  decode(m, out, b, z, y, x);
  const int D2 = out.D * 2, H2 = out.H * 2, W2 = out.W * 2;
  float g[8] = {};
  add_oct(g, ld_oct(gout.p + m * gout.cs + gout.co + c));
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long sv = (((long long)b * D2 + 2 * z + (q >> 2)) * H2 + 2 * y + ((q >> 1) & 1)) * W2 + 2 * x + (q & 1);
    bf16* d = gin.p + sv * gin.cs + gin.co + c;
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = 0.125f * g[u];
    if (accumulate) add_oct(v, ld_oct(d));   // the old value plus the new one: the sum of two is the same either way round
    Oct r;
#pragma unroll
    for (int u = 0; u < 4; ++u) r.h[u] = __floats2bfloat162_rn(v[2 * u], v[2 * u + 1]);
    st_oct(d, r);
  }
}

// nearest-neighbour upsampling x2: fine voxel takes its parent's value.
__global__ void k_up_fwd(Vol fine, int C, Act in, Act o) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int no = C >> 3;
  if (e >= fine.voxels() * no) return;
  const long long m = e / no;
  const int c = 8 * (int)(e - m * no);
  int b, z, y, x;
  decode(m, fine, b, z, y, x);
  const long long pv = (((long long)b * (fine.D / 2) + z / 2) * (fine.H / 2) + y / 2) * (fine.W / 2) + x / 2;
  st_oct(o.p + m * o.cs + o.co + c, ld_oct(in.p + pv * in.cs + in.co + c));
}

// parent gradient = sum of its eight children's gradients.
__global__ void k_up_bwd(Vol coarse, int C, Act gfine, Act gout) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int no = C >> 3;
  if (e >= coarse.voxels() * no) return;
  const long long m = e / no;
  const int c = 8 * (int)(e - m * no);
  int b, z, y, x;
  decode(m, coarse, b, z, y, x);
  const int D2 = coarse.D * 2, H2 = coarse.H * 2, W2 = coarse.W * 2;
  float s[8] = {};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long sv = (((long long)b * D2 + 2 * z + (q >> 2)) * H2 + 2 * y + ((q >> 1) & 1)) * W2 + 2 * x + (q & 1);
    add_oct(s, ld_oct(gfine.p + sv * gfine.cs + gfine.co + c));
  }
  Oct r;
#pragma unroll
  for (int q = 0; q < 4; ++q) r.h[q] = __floats2bfloat162_rn(s[2 * q], s[2 * q + 1]);
  st_oct(gout.p + m * gout.cs + gout.co + c, r);
}

// 1x1 head: out[v] = sum_c w[c] * in[v][c] + b   (FP32 output)
__global__ void k_head_fwd(long long M, int C, Act in, const float* __restrict__ w, float* __restrict__ out) {
  const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  float s = w[C];
  for (int c = 0; c < C; ++c) s = fmaf(w[c], __bfloat162float(in.p[m * in.cs + in.co + c]), s);
  out[m] = s;
}

// gin[v][c] = gout[v] * w[c]; dw[c] += sum_v gout[v] * in[v][c]; dw[C] += sum_v gout[v], C = 16.
// Each thread sums over its voxels in registers, the block once at the end (shared-memory
// atomics per voxel took 83 us at 262,144).
constexpr int kHeadC = 16;
__global__ void __launch_bounds__(256) k_head_bwd(long long M, Act in, const float* __restrict__ w,
                                                  const float* __restrict__ gout, Act gin, float* __restrict__ dw) {
  __shared__ float s[8][kHeadC + 1];
  float a[kHeadC + 1] = {};
  for (long long m = (long long)blockIdx.x * 256 + threadIdx.x; m < M; m += (long long)gridDim.x * 256) {
    const float g = gout[m];
#pragma unroll
    for (int c = 0; c < kHeadC; c += 8) {
      float x[8] = {};
      add_oct(x, ld_oct(in.p + m * in.cs + in.co + c));
      Oct r;
#pragma unroll
      for (int q = 0; q < 4; ++q) r.h[q] = __floats2bfloat162_rn(g * w[c + 2 * q], g * w[c + 2 * q + 1]);
      st_oct(gin.p + m * gin.cs + gin.co + c, r);
#pragma unroll
      for (int q = 0; q < 8; ++q) a[c + q] += g * x[q];
    }
    a[kHeadC] += g;
  }
#pragma unroll
  for (int c = 0; c <= kHeadC; ++c) {
    for (int d = 16; d > 0; d >>= 1) a[c] += __shfl_xor_sync(0xffffffffu, a[c], d);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5][c] = a[c];
  }
  __syncthreads();
  if (threadIdx.x <= kHeadC) {
    float x = 0.f;
    for (int q = 0; q < 8; ++q) x += s[q][threadIdx.x];
    atomicAdd(&dw[threadIdx.x], x);
  }
}

// mean squared error: g = 2 (out - t) / M, loss += sum (out - t)^2 / M
__global__ void __launch_bounds__(256) k_mse(long long M, const float* __restrict__ out, const float* __restrict__ t,
                                             float* __restrict__ g, double* loss) {
  __shared__ double s[8];
  double a = 0.0;   // FP32 squares, added in FP64: a thread's voxels grow with the batch
  for (long long m = (long long)blockIdx.x * 256 + threadIdx.x; m < M; m += (long long)gridDim.x * 256) {
    const float d = out[m] - t[m];
    g[m] = 2.f * d / (float)M;
    a += (double)(d * d);
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < 8; ++q) a += s[q];
    if (a != 0.0) atomicAdd(loss, a / (double)M);
  }
}

// Adam (FP32 master weights) and the BF16 copies the kernels read: the forward
// layout [n][tap][k] and the transposed input-gradient layout [k][tap][n].
__global__ void k_adam(int n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, float lr, float b1, float b2, float c1, float c2, float eps) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float gg = g[e];
  const float a = b1 * m1[e] + (1.f - b1) * gg;
  const float b = b2 * m2[e] + (1.f - b2) * gg * gg;
  m1[e] = a;
  m2[e] = b;
  p[e] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
}

__global__ void k_cast_conv_weights(int N, int K, const float* __restrict__ w, bf16* __restrict__ wf,
                                    bf16* __restrict__ wt) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= N * 27 * K) return;
  const int k = e % K, tap = (e / K) % 27, n = e / (27 * K);
  const bf16 v = __float2bfloat16(w[e]);
  wf[e] = v;
  wt[((size_t)k * 27 + tap) * N + n] = v;
}

// ------------------------------------------------------------ launch helpers

// The most dynamic shared memory of a launch, and every kernel's limit: the limit belongs to the
// kernel, so one set to a launch's own size could have another thread's launch refused.
constexpr size_t kSmemMax = 227 * 1024 - 512;
constexpr int kSms = 152;

// Blocks of 128 R entries and the rings' depths: the largest R that leaves two blocks per SM
// (fewer entries are loaded twice), then as many buffers as two blocks per SM, or one, hold.
template <int N>
void launch_conv3(cudaStream_t st, const Vol& vol, Act X, int K, const bf16* W, const float* bias, int relu, int sign,
                  Act Y, int* err) {
  const Seq seq = make_seq(vol);
  const size_t wstep = (size_t)3 * K * N * 2;
  auto run = [&](int R) { return (size_t)(128 * R + 2 * (seq.Wp + 1)) * K * 2; };
  auto blocks = [&](int R) { return (seq.n + 128 * R - 1) / (128 * R); };
  int R = 4;
  while (R > 1 && (R * N > 256 || blocks(R) < 2 * kSms || 3 * run(R) + 3 * wstep > kSmemMax / 2)) R >>= 1;
  int NX = 3, NB = 9;
  const size_t cap = 3 * run(R) + 2 * wstep <= kSmemMax / 2 ? kSmemMax / 2 : kSmemMax;
  while (NX > 1 && NX * run(R) + 2 * wstep > cap) --NX;
  while (NB > 2 && NX * run(R) + NB * wstep > cap) --NB;
  const size_t smem = NX * run(R) + NB * wstep;
  if (smem > kSmemMax || seq.n >= (1ll << 31)) {   // no network layer of this library (K <= 96, strips) gets here
    cudaMemsetAsync(err, 1, sizeof(int), st);
    return;
  }
  cudaFuncSetAttribute(k_conv3<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  k_conv3<N><<<(unsigned)blocks(R), kConvThreads, smem, st>>>(seq, X, K, W, bias, relu, sign, Y, R, NX, NB, err);
}

void conv(cudaStream_t st, const Vol& vol, Act X, int K, const bf16* W, const float* bias, int relu, int sign, Act Y,
          int N, int* err) {
  switch (N) {
    case 16: launch_conv3<16>(st, vol, X, K, W, bias, relu, sign, Y, err); break;
    case 32: launch_conv3<32>(st, vol, X, K, W, bias, relu, sign, Y, err); break;
    case 48: launch_conv3<48>(st, vol, X, K, W, bias, relu, sign, Y, err); break;
    case 64: launch_conv3<64>(st, vol, X, K, W, bias, relu, sign, Y, err); break;
    case 96: launch_conv3<96>(st, vol, X, K, W, bias, relu, sign, Y, err); break;
    default: break;
  }
}

namespace {
// The shape of a k_wgrad_tc launch; stages 0 where the tensor-core form does not fit.
struct WgradShape {
  int nz, pairs, gx, gy, stages;
  size_t smem;
};
WgradShape wgrad_shape(const Seq& seq, int N, int K) {
  WgradShape w{};
  // all three planes of a pair in one MMA (at most 256 columns) where two stages of them fit
  const size_t run = (size_t)(128 + 2 * (seq.Wp + 1)) * K * 2, line = 8 * 128 * 16;
  w.nz = 3 * K <= 256 && 2 * (3 * run + line) <= kSmemMax ? 3 : 1;
  const int most = std::min(9, 512 / (w.nz * K)), groups = (9 + most - 1) / most;
  w.pairs = (9 + groups - 1) / groups;
  const size_t stage = w.nz * run + line;
  w.stages = (int)std::min<size_t>(kMaxStagesW, kSmemMax / stage);
  if (N > 64 || N % 16 != 0 || w.stages < 2 || seq.n >= (1ll << 31)) w.stages = 0;
  w.smem = w.stages * stage;
  w.gx = groups * (3 / w.nz);
  w.gy = (int)std::max(1ll, std::min((seq.n + 127) / 128, (long long)(kSms / w.gx)));
  return w;
}
}  // namespace

size_t wgrad_workspace(const Vol& vol, int N, int K) {
  const WgradShape w = wgrad_shape(make_seq(vol), N, K);
  return w.stages ? (size_t)w.gy * N * 27 * K : 0;
}

void wgrad(cudaStream_t st, const Vol& vol, Act dZ, int N, Act X, int K, float* dW, float* work, int* err) {
  const Seq seq = make_seq(vol);
  const WgradShape w = wgrad_shape(seq, N, K);
  if (!w.stages) {
    wgrad_cuda_cores(st, vol, dZ, N, X, K, dW);
    return;
  }
  cudaFuncSetAttribute(k_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  k_wgrad_tc<<<dim3((unsigned)w.gx, (unsigned)w.gy), kConvThreads, w.smem, st>>>(seq, dZ, N, X, K, work, w.nz, w.pairs,
                                                                                 w.stages, err);
  const int n = N * 27 * K;
  k_wgrad_sum<<<(unsigned)((n / 4 + 31) / 32), 256, 0, st>>>(work, n, w.gy, dW);
}

void wgrad_cuda_cores(cudaStream_t st, const Vol& vol, Act dZ, int N, Act X, int K, float* dW) {
  const long long M = vol.voxels();
  const long long chunk = 4096;
  dim3 grid((unsigned)((M + chunk - 1) / chunk), 27);
  const size_t smem = (size_t)kWgTile * (N + K) * sizeof(float);
  k_wgrad<<<grid, 256, smem, st>>>(vol, dZ, N, X, K, dW, chunk);
}

static unsigned strided_blocks(long long threads) {   // a few blocks per SM, each thread several elements
  return (unsigned)std::max(1ll, std::min((threads + 255) / 256, 4ll * kSms));
}

void relu_bias_bwd(cudaStream_t st, long long M, int N, Act dY, Act Y, float* db) {
  k_relu_bias_bwd<<<strided_blocks(M * (N / 8)), 256, 0, st>>>(M, N, dY, Y, db);
}

void pool_fwd(cudaStream_t st, const Vol& out, int C, Act in, Act o) {
  k_pool_fwd<<<(unsigned)((out.voxels() * (C / 8) + 255) / 256), 256, 0, st>>>(out, C, in, o);
}

void pool_bwd(cudaStream_t st, const Vol& out, int C, Act gout, Act gin, int accumulate) {
  k_pool_bwd<<<(unsigned)((out.voxels() * (C / 8) + 255) / 256), 256, 0, st>>>(out, C, gout, gin, accumulate);
}

void up_fwd(cudaStream_t st, const Vol& fine, int C, Act in, Act o) {
  k_up_fwd<<<(unsigned)((fine.voxels() * (C / 8) + 255) / 256), 256, 0, st>>>(fine, C, in, o);
}

void up_bwd(cudaStream_t st, const Vol& coarse, int C, Act gfine, Act gout) {
  k_up_bwd<<<(unsigned)((coarse.voxels() * (C / 8) + 255) / 256), 256, 0, st>>>(coarse, C, gfine, gout);
}

void head_fwd(cudaStream_t st, long long M, int C, Act in, const float* w, float* out) {
  k_head_fwd<<<(unsigned)((M + 255) / 256), 256, 0, st>>>(M, C, in, w, out);
}

void head_bwd(cudaStream_t st, long long M, Act in, const float* w, const float* gout, Act gin, float* dw) {
  k_head_bwd<<<strided_blocks(M), 256, 0, st>>>(M, in, w, gout, gin, dw);
}

void mse(cudaStream_t st, long long M, const float* out, const float* t, float* g, double* loss) {
  k_mse<<<strided_blocks(M), 256, 0, st>>>(M, out, t, g, loss);
}

void adam(cudaStream_t st, int n, float* p, const float* g, float* m1, float* m2, float lr, int step) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<(n + 255) / 256, 256, 0, st>>>(n, p, g, m1, m2, lr, b1, b2, c1, c2, 1e-8f);
}

void cast_conv_weights(cudaStream_t st, int N, int K, const float* w, bf16* wf, bf16* wt) {
  k_cast_conv_weights<<<(N * 27 * K + 255) / 256, 256, 0, st>>>(N, K, w, wf, wt);
}

}  // namespace unet
}  // namespace ib3d
