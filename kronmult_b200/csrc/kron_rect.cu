// Rectangular factors, one shape for the whole batch (the vbatched calls, and
// square sizes without a kernel of their own), FP64, vectors that fit shared
// memory.
//
// A group of GS threads works through a contiguous, balanced range of
// entries.  The next entry's factors and vector are on their way to shared
// memory (cp.async) while the current one is computed, and the pointers of
// the one after next on their way to the group's slots, so no dependent round
// trip stalls the group; the mode products follow a list of steps computed on
// the host (kron_rect.cuh).  Results go into y by red.global.add (one add per
// element: exclusive outputs get the plain sum, aliasing ones add up).
//
// (kronmult_vbatched.hpp:17-228 copies x to scratch and runs one 64-thread
// block per entry through global memory.)
//
// 4096 entries of 576 elements (60 MB): 94 -> 30 us, of which HBM alone would
// take 9; fifteen warps an SM that wait for the steps' latencies are the bound
// now (an instruction in 34% of a scheduler's cycles, the shared-memory pipe
// 31% busy).  Before, two
// groups a block worked through runs of eight entries in series, recomputing
// every step's shape, dividing per fibre, and waiting out each load.
#include <algorithm>
#include <cstdint>

#include "kron_launch.h"
#include "kron_ptx.cuh"
#include "kron_rect.cuh"

namespace kron {

namespace {

using namespace ptx;

constexpr int RECT_THREADS = 256, RECT_WIDE = 512;

struct RectArgs
{
  RectStep st[MAXD];
  int nin, nout, asz;   // elements of x, y and all factors
  int buf;              // elements of a vector buffer (even)
  int group;            // elements of a group's shared memory
  int GS;
};

__device__ __forceinline__ void cp8(double *dst, const double *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}

// AREG, MINB: elements of a factor held in registers, blocks per SM
template <int THREADS, int AREG, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
    kron_rect_kernel(const __grid_constant__ Params p, const __grid_constant__ RectArgs r)
{
  extern __shared__ __align__(16) double smem[];
  __shared__ const double *s_ptr[8][3][8]; // per group: pointers of three entries
  const int GS = r.GS;
  const int ng = THREADS / GS, g = threadIdx.x / GS, t = threadIdx.x - g * GS;
  double *base = smem + (size_t)g * r.group;
  int e, ee;
  group_range(p, blockIdx.x * ng + g, gridDim.x * ng, e, ee);
  if (e >= ee)
    return;
  const int d = p.d;

  // pointer j of position e: A_1..A_d, x at 6, y at 7
  auto pointer = [&](int e, int j) -> const double * {
    const int k = entry_index(p, e);
    if (j < 6)
    {
      if (j >= d)
        return nullptr;
      if (p.layout == LAYOUT_BATCHED || p.layout == LAYOUT_PBATCHED)
        return static_cast<const double *>(p.A) + ((long long)k * d + j) * p.n[0] * p.n[0];
      return static_cast<const double *>(p.pA[(long long)k * p.apk + j]);
    }
    if (p.layout == LAYOUT_BATCHED)
      return j == 6 ? static_cast<const double *>(p.X) + (long long)k * p.xstride
                    : static_cast<const double *>(p.Y) + (long long)k * p.ystride;
    return static_cast<const double *>(j == 6 ? p.pX[k] : p.pY[k]);
  };
  // vector and factors of the entry whose pointers are in `ptr`
  const int warp = t >> 5, lane = t & 31, nw = GS >> 5;
  auto issue = [&](const double *const *ptr, int b) {
    double *x       = base + b * r.buf;
    double *as      = base + 3 * r.buf + b * ((r.asz + 1) & ~1);
    const double *s = ptr[6];
    if (aligned16(s))
    {
      for (int u = t; u < r.nin / 2; u += GS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(x + 2 * u)),
                     "l"(s + 2 * u)
                     : "memory");
      if ((r.nin & 1) && t == 0)
        cp8(x + r.nin - 1, s + r.nin - 1);
    }
    else
      for (int u = t; u < r.nin; u += GS)
        cp8(x + u, s + u);
    int o = 0;
    for (int q = 0; q < d; q++)
    {
      const int mq = r.st[q].mq, sz = mq * r.st[q].nq, l = r.st[q].mode;
      if (q % nw == warp)
      {
        const int ld = p.layout == LAYOUT_XBATCHED ? p.lda : mq;
        for (int u = lane; u < sz; u += 32)
          cp8(as + o + u, ld == mq ? ptr[l] + u
                                   : ptr[l] + u % mq + (long long)(u / mq) * ld);
      }
      o += sz;
    }
  };

  if (t < 8)
  {
    s_ptr[g][0][t] = pointer(e, t);
    if (e + 1 < ee)
      s_ptr[g][1][t] = pointer(e + 1, t);
  }
  group_sync(g, GS);
  issue(s_ptr[g][0], 0);
  for (int i = 0;; i++)
  {
    const int b     = i & 1;
    const bool more = e + 1 < ee;
    asm volatile("cp.async.wait_all;" ::: "memory");
    group_sync(g, GS);
    const double *pn = nullptr;
    if (more)
    {
      issue(s_ptr[g][(i + 1) % 3], b ^ 1);
      if (t < 8 && e + 2 < ee)
        pn = pointer(e + 2, t);
    }
    // the vector's stage is one of the two buffers, the third the other
    double *cur = base + b * r.buf, *nxt = base + 2 * r.buf;
    rect_modes<double, AREG, true>(r.st, d, 1, cur, nxt, base + 3 * r.buf + b * ((r.asz + 1) & ~1), t, GS, g);
    double *y = const_cast<double *>(s_ptr[g][i % 3][7]);
    for (int q = t; q < r.nout; q += GS)
      red_add(y + q, cur[q]);
    if (!more)
      break;
    if (t < 8 && e + 2 < ee)
      s_ptr[g][(i + 2) % 3][t] = pn;
    ++e;
  }
}

// Threads an entry, by its largest intermediate: about a dozen elements a
// thread in each step, so that the fixed work of a step (its list entry, the
// factor, a barrier) is spread over several fibres.  Microseconds with 32 / 64
// / 128 threads: 150 elements (30000 entries) 62 / 105 / 186, 1152 elements
// (4096 entries) 33 / 31 / 39, 1536 elements (5000 entries) - / 76 / 66.
int rect_group_size(long long elems)
{
  return elems >= 4096 ? 256 : elems >= 1280 ? 128 : elems >= 512 ? 64 : 32;
}

// elements of a group's shared memory
bool rect_args(const Params &p, RectArgs &r)
{
  const bool fwd = choose_forward(p.d, p.m, p.n);
  const long long mi = max_intermediate(p.d, p.m, p.n, fwd);
  if (mi * 8 > device_info().max_smem_optin)
    return false;
  for (int l = 0; l < p.d; l++)
    if (p.m[l] > 255 || p.n[l] > 255)
      return false;
  rect_plan(r.st, p.d, p.m, p.n, 0, fwd, 1);
  long long nin = 1, nout = 1, asz = 0;
  for (int l = 0; l < p.d; l++)
  {
    nin *= p.n[l];
    nout *= p.m[l];
    asz += (long long)p.m[l] * p.n[l];
  }
  r.nin = (int)nin;
  r.nout = (int)nout;
  r.asz = (int)asz;
  r.buf = (int)((mi + 1) & ~1LL);
  const long long group = 3LL * r.buf + 2 * ((asz + 1) & ~1LL);
  if (group * 8 > device_info().max_smem_optin)
    return false;
  r.group = (int)group;
  r.GS    = rect_group_size(mi);
  return true;
}

} // namespace

bool rect_supported(const Params &p, int prec)
{
  return prec == PREC_F64 && !p.seg_off && (p.accum == ACC_DISTINCT || p.accum == ACC_ATOMIC);
}

int launch_rect(const Params &p, cudaStream_t stream)
{
  if (p.eend <= p.ebase)
    return KRON_SUCCESS;
  RectArgs r{};
  if (!rect_args(p, r))
    return KRON_ERROR_NOT_SUPPORTED;
  // short vectors: three blocks an SM and factors of up to 16 elements in
  // registers (80 a thread); longer ones reuse a factor over more fibres and
  // gain from holding up to 36 (two blocks; 576 elements: 31 against 35 us,
  // 96 elements: 42 against 50 us the other way)
  const void *fn = r.buf < 512
                       ? reinterpret_cast<const void *>(&kron_rect_kernel<RECT_THREADS, 16, 3>)
                       : reinterpret_cast<const void *>(&kron_rect_kernel<RECT_THREADS, 36, 2>);
  // as many groups a block as its threads and half an SM's shared memory give
  // (1 KB a block is the hardware's, 2 KB hold the kernel's own variables), at
  // least one: groups twice as large are faster than one block an SM (square d =
  // 2, n = 16, 5000 entries of 14 KB: 33 against 51 us; d = 3, n = 13, 3000 of 61
  // KB: 197 against 260); an entry an SM takes twice the threads (d = 3, n = 18,
  // 2000 entries of 156 KB: 426 against 582 us)
  const long long half = device_info().smem_per_sm / 2 - 3072, need = r.group * 8LL;
  if (need > device_info().max_smem_optin - 2048)
    return KRON_ERROR_NOT_SUPPORTED;
  while (r.GS < RECT_THREADS && RECT_THREADS / r.GS * need > half)
    r.GS *= 2;
  int threads = RECT_THREADS;
  if (need > half)
  {
    fn      = reinterpret_cast<const void *>(&kron_rect_kernel<RECT_WIDE, 36, 1>);
    threads = r.GS = RECT_WIDE;
  }
  const int ng      = threads / r.GS;
  const size_t smem = (size_t)ng * r.group * 8;
  int per_sm        = 1;
  if (cached_occupancy(fn, threads, smem, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  const long long work = (long long)p.eend - p.ebase;
  const long long grid =
      std::min<long long>((work + ng - 1) / ng, (long long)device_info().sms * per_sm);
  Params pp    = p;
  void *args[] = {&pp, &r};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(threads), args, smem, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

} // namespace kron
