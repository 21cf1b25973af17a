// Resident kernel: FP32 vectors of square d = 6, n = 6 (187 KB) held whole in one
// block's shared memory.  No workspace, x read once, y added once.
//
// x is viewed as 36 rows (i_1, i_2) of 1296 contiguous elements, which arrive
// by TMA bulk copies.  Three register-blocked passes of two modes, a thread
// holding a fibre of 36 elements and one 6x6 factor at a time:
//   pass A  modes 5, 6 in place on contiguous fibres, as their rows arrive;
//   pass B  modes 3, 4 in place on strided fibres;
//   pass C  modes 1, 2 on the 1296 columns, results added into y from
//           registers (red.global.add).
// The last warp has no columns in the last round: when the other warps have
// read theirs it starts the next entry's copies, so the rows (prefetched into
// L2 an entry ahead) land while the block still multiplies and adds.
//
// Contiguous fibres are 9 16-byte units apart, so the 16-byte accesses of
// eight neighbouring lanes fall on distinct banks; strided fibres and columns
// are read by consecutive lanes at consecutive addresses.
//
// 448 threads: 1296 fibres in three rounds, and 128 registers a thread hold a
// fibre, a factor and the loop without spills (16 warps would need as many
// rounds, 20 warps leave 96 registers).
//
// Every mbarrier wait is bounded (wait_limit() polls).  A block whose copies
// do not arrive in time records 1 in the device status word, lets them land
// (bounded by drain_limit()), stops writing y and issuing copies, and leaves.
//
// Bound by HBM at best (2.3 GB for 4096 entries: 0.35 ms); measured 0.491 ms
// (72% of the measured copy bandwidth) against 0.939 ms for the slab-cluster
// kernel, whose seven active warps an SM spend half their time at cluster
// barriers and on remote shared-memory reads.
//
// The product is the reference's (kronmult6_batched.hpp:41-75, computed there
// by kronmultv_recur.hpp:117-145).
#include <algorithm>
#include <cstdint>

#include "kron_fibre.cuh"
#include "kron_launch.h"
#include "kron_ptx.cuh"

namespace kron {

namespace {

using namespace ptx;

constexpr int RS_N = 6, RS_N2 = 36, RS_LT = 1296;
constexpr int RS_ROWS    = RS_N2;
constexpr int RS_FIB     = RS_LT; // fibres of passes A and B, columns of pass C
constexpr int RS_THREADS = 448;
constexpr int RS_RND     = (RS_FIB + RS_THREADS - 1) / RS_THREADS;
static_assert(RS_RND * RS_THREADS - 32 >= RS_FIB, "the last round leaves a warp to spare");
// rows arrive in groups, each with its own mbarrier
constexpr int RS_GROWS = 6, RS_GROUPS = RS_ROWS / RS_GROWS, RS_GLEN = RS_GROWS * RS_LT;
constexpr int RS_ASZ = 6 * RS_N2;
constexpr size_t RS_OFF_A = 128;
constexpr size_t RS_OFF_X = RS_OFF_A + (2 * RS_ASZ * sizeof(float) + 127) / 128 * 128;
constexpr size_t RS_SMEM  = RS_OFF_X + (size_t)RS_ROWS * RS_LT * sizeof(float);

__global__ void __launch_bounds__(RS_THREADS, 1)
    kron_resident_kernel(const __grid_constant__ Params p, int *status, long long spin,
                         long long drain)
{
  using T         = float;
  constexpr int N = RS_N, N2 = RS_N2, LT = RS_LT;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  T *xs          = reinterpret_cast<T *>(smem + RS_OFF_X);
  auto stage_a   = [&](int b) { return reinterpret_cast<T *>(smem + RS_OFF_A) + b * RS_ASZ; };
  const int tid  = threadIdx.x;
  const long long tot = p.eend - p.ebase;
  const int eb = p.ebase + (int)(tot * blockIdx.x / gridDim.x);
  const int ee = p.ebase + (int)(tot * (blockIdx.x + 1) / gridDim.x);
  if (eb >= ee)
    return;
  uint64_t stream;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(stream));

  auto entry_x = [&](int e) {
    const int k = entry_index(p, e);
    return p.layout == LAYOUT_BATCHED ? static_cast<const T *>(p.X) + (long long)k * p.xstride
                                      : static_cast<const T *>(p.pX[k]);
  };
  // this thread's factor element of position e into `as` (tid < RS_ASZ)
  auto load_a = [&](int e, T *as) {
    const int k = entry_index(p, e), l = tid / N2, ij = tid - l * N2;
    const T *src;
    if (p.layout == LAYOUT_BATCHED || p.layout == LAYOUT_PBATCHED)
      src = static_cast<const T *>(p.A) + (long long)k * RS_ASZ + tid;
    else
    {
      const int ld = p.layout == LAYOUT_XBATCHED ? p.lda : N;
      src          = static_cast<const T *>(p.pA[(long long)k * p.apk + l]) + ij % N +
            (long long)(ij / N) * ld;
    }
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(as + tid)), "l"(src)
                 : "memory");
  };
  // one warp: start the copies of position e's rows (none when x is not 16-byte
  // aligned: pass A then loads them)
  auto issue = [&](int e) {
    const T *x     = entry_x(e);
    const bool ok  = aligned16(x);
    const int lane = tid & 31;
    if (lane < RS_GROUPS)
    {
      mbar_expect_tx(&bars[lane], ok ? RS_GLEN * (unsigned)sizeof(T) : 0u);
      if (ok)
        tma_load_1d(xs + lane * RS_GLEN, x + lane * RS_GLEN, RS_GLEN * (unsigned)sizeof(T),
                    &bars[lane]);
    }
  };

  if (tid == 0)
  {
    for (int g = 0; g < RS_GROUPS; g++)
      mbar_init(&bars[g], 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (tid < 32)
    issue(eb);
  if (tid < RS_ASZ)
    load_a(eb, stage_a(0));
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  unsigned parity = 0;
  for (int e = eb; e < ee; ++e)
  {
    const int b     = (e - eb) & 1;
    const T *as     = stage_a(b);
    const bool more = e + 1 < ee;
    if (more && tid >= RS_THREADS - 32 && (tid & 31) < RS_GROUPS)
    {
      const T *x = entry_x(e + 1) + (tid & 31) * RS_GLEN;
      if (aligned16(x))
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x),
                     "r"(RS_GLEN * (unsigned)sizeof(T))
                     : "memory");
    }

    // ---- pass A: modes 5 and 6, contiguous fibres, as their rows arrive
    bool ok = true;
    if (!aligned16(entry_x(e))) // block-uniform
    {
      // the phase completes (without a copy) when the rows may be overwritten
      ok = mbar_wait_bounded(&bars[0], parity, spin);
      const T *x = entry_x(e);
      for (int i = tid; ok && i < RS_ROWS * LT; i += RS_THREADS)
        xs[i] = __ldg(x + i);
      __syncthreads();
    }
#pragma unroll 1
    for (int f = tid; f < RS_FIB; f += RS_THREADS)
    {
      ok   = ok && mbar_wait_bounded(&bars[f / (RS_GROWS * N2)], parity, spin);
      T *c = xs + f * N2;
      T v[N2];
      load_chunk<T, N>(c, v);
      apply_fast<T, N>(v, as + 5 * N2);
      apply_slow<T, N>(v, as + 4 * N2);
      store_chunk<T, N>(c, v);
    }
    if (!__syncthreads_and(ok))
    {
      if (tid == 0)
      {
        if (status)
          atomicExch(status, 1);
        for (int g = 0; g < RS_GROUPS; g++)
          mbar_wait_bounded(&bars[g], parity, drain);
      }
      return;
    }
    parity ^= 1;
    // every warp is past the last entry's pass C, which read this stage
    if (more && tid < RS_ASZ)
      load_a(e + 1, stage_a(b ^ 1));
    // ---- pass B: modes 3 and 4, strided fibres
#pragma unroll 1
    for (int f = tid; f < RS_FIB; f += RS_THREADS)
    {
      const int row = f / N2;
      T *c          = xs + row * LT + (f - row * N2);
      T v[N2];
#pragma unroll
      for (int q = 0; q < N2; q++)
        v[q] = c[q * N2];
      apply_fast<T, N>(v, as + 3 * N2);
      apply_slow<T, N>(v, as + 2 * N2);
#pragma unroll
      for (int q = 0; q < N2; q++)
        c[q * N2] = v[q];
    }
    asm volatile("cp.async.wait_all;" ::: "memory"); // the next factors
    __syncthreads();

    // ---- pass C: modes 1 and 2 on columns, added into y
    T *y = entry_y<T>(p, entry_index(p, e));
#pragma unroll 1
    for (int r = 0; r < RS_RND; r++)
    {
      const int f     = tid + r * RS_THREADS;
      const bool last = r == RS_RND - 1;
      if (last && tid >= RS_THREADS - 32)
      {
        fence_proxy_async();
        asm volatile("bar.sync 1, %0;" ::"n"(RS_THREADS) : "memory");
        if (more)
          issue(e + 1);
        break;
      }
      const bool have = f < RS_FIB;
      T v[N2];
      if (have)
      {
#pragma unroll
        for (int q = 0; q < N2; q++)
          v[q] = xs[q * LT + f];
      }
      if (last)
      {
        // this thread is done with the rows; its accesses come before the
        // copies that overwrite them
        fence_proxy_async();
        asm volatile("bar.arrive 1, %0;" ::"n"(RS_THREADS) : "memory");
      }
      if (have)
      {
        apply_fast<T, N>(v, as + 1 * N2);
        apply_slow<T, N>(v, as + 0 * N2);
#pragma unroll
        for (int q = 0; q < N2; q++)
          asm volatile("red.global.add.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(y + (long long)q * LT + f),
                       "f"(v[q]), "l"(stream)
                       : "memory");
      }
    }
  }
}

} // namespace

bool resident_supported(const Params &p, int prec)
{
  if (prec != PREC_F32 || p.seg_off || (p.accum != ACC_DISTINCT && p.accum != ACC_ATOMIC) ||
      p.d != 6)
    return false;
  for (int l = 0; l < 6; l++)
    if (p.m[l] != 6 || p.n[l] != 6)
      return false;
  return true;
}

int launch_resident(const Params &p, cudaStream_t stream)
{
  if (p.eend <= p.ebase)
    return KRON_SUCCESS;
  const void *fn = reinterpret_cast<const void *>(&kron_resident_kernel);
  if (RS_SMEM > (size_t)device_info().max_smem_optin)
    return KRON_ERROR_NOT_SUPPORTED;
  int per_sm = 1;
  if (cached_occupancy(fn, RS_THREADS, RS_SMEM, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  const int grid = std::min(device_info().sms, p.eend - p.ebase);
  Params pp      = p;
  int *status    = device_status_ptr();
  long long sp   = wait_limit();
  long long dr   = drain_limit();
  void *args[]   = {&pp, &status, &sp, &dr};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(RS_THREADS), args, RS_SMEM, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

} // namespace kron
