// Pair kernel: square vectors of d = 4..6 modes that fit one block's shared
// memory, a thread a fibre of two modes (n^2 elements) in registers, FP64 and
// FP32, every layout and accumulation mode.
//
// The square and the pipelined kernels applied one mode a pass: each pass
// moves the vector through shared memory once, n = 7 and 8 reading the factor
// from there at every product, and the square kernel waited out every entry's
// pointers and operands.  Here a block (one thread a fibre where F = n^(d-2)
// allows) works through a contiguous, balanced range of entries in d / 2
// passes:
//   modes 1, 2 on strided fibres, modes 3, 4 (d = 6; d = 5: between them and
//   the last), the last two (d = 5: the last) on contiguous fibres.
// The next entry's operands are on their way by cp.async (where two vectors
// fit; else its x is prefetched into L2) and the pointers of the one after
// next on their way to registers.  Fibres lie padded to an odd number of
// 16-byte units (even n; odd n needs no padding), so that neighbouring lanes'
// 16-byte accesses hit distinct banks.  A factor is read column by column, 16
// bytes at a time, for RB rows of the fibre: the fibre, RB rows of results and
// a column are what a thread holds.
//
// Modes go in the square kernel's order and each result is the same chain of
// fma, so exclusive outputs are the same bit for bit.  Results of consecutive
// entries with one output are summed in shared memory (each thread its own
// fibre) and added once, by red.global.add; FP32 (exclusive outputs only) goes
// through a load, an add and a store: an FP32 add in the L2 cache would flush
// subnormals.
//
// Bound by latency with few warps an SM (n = 8: six, by shared memory and
// registers; an instruction in 26% of a scheduler's cycles; FP64 d = 4, n = 8
// spills 176 bytes a thread, 146 with sums in shared memory, d = 5, n = 7 300):
// batched FP64, before and after, d = 4, n = 8, 6000
// entries 324 -> 165 us (0.60 GB, HBM alone 92); d = 5, n = 7, 1000 entries 312
// -> 129 (62); d = 6, n = 3, 10000 entries 132 -> 47 (27); 7200 entries of d = 4,
// n = 8 on 800 outputs 332 -> 163; 36000 of d = 4, n = 5 on 4000 360 -> 89.
//
// (kronmultv_recur.hpp:117-145 computes the same products, a block an entry
// through global memory.)
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kron_fibre.cuh"
#include "kron_launch.h"
#include "kron_ptx.cuh"

namespace kron {

namespace {

using namespace ptx;

template <typename T, int D, int N, bool MERGE>
struct PairShape
{
  static constexpr int N2 = N * N, L = cpow(N, D), F = L / N2;
  static constexpr int V  = 16 / (int)sizeof(T);
  static constexpr bool VEC = N % 2 == 0; // fibres are whole 16-byte units
  static constexpr int CS   = N2 + (VEC && N2 / V % 2 == 0 ? V : 0);
  static constexpr int XLEN = (F * CS + V - 1) / V * V;
  static constexpr int LD   = (N + V - 1) / V * V; // of a staged factor
  static constexpr int AF   = N * LD;
  static constexpr int ROUNDS  = (F + 351) / 352;
  static constexpr int THREADS = ((F + ROUNDS - 1) / ROUNDS + 31) / 32 * 32;
  // rows of a fibre whose results are computed at a time
  static constexpr int RB = sizeof(T) == 8 ? (N == 8 ? 2 : N == 7 ? 4 : N == 6 ? 3 : N) : (N == 8 ? 4 : N);
  static constexpr size_t bytes(int stages)
  {
    return ((size_t)XLEN * (stages + (MERGE ? 1 : 0)) + 2 * D * AF) * sizeof(T);
  }
  static constexpr int STAGES  = bytes(2) <= 220 * 1024 ? 2 : 1;
  static constexpr size_t SMEM = bytes(STAGES);
  __device__ static constexpr int pos(int i) { return i / N2 * CS + i % N2; }
};

// A (column stride LD) along the faster (FAST) or the slower mode of v
template <typename T, int N, int LD, int RB, bool FAST>
__device__ __forceinline__ void pair_apply(T (&v)[N * N], const T *A)
{
  constexpr int V = 16 / (int)sizeof(T);
  using VT        = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
#pragma unroll
  for (int r0 = 0; r0 < N; r0 += RB)
  {
    T w[RB][N];
#pragma unroll
    for (int j = 0; j < N; j++)
    {
      T a[LD];
#pragma unroll
      for (int u = 0; u < LD; u += V)
      {
        const VT q = *reinterpret_cast<const VT *>(A + j * LD + u);
        a[u]       = q.x;
        a[u + 1]   = q.y;
        if constexpr (V == 4)
        {
          a[u + 2] = q.z;
          a[u + 3] = q.w;
        }
      }
#pragma unroll
      for (int r = 0; r < RB; r++)
        if (r0 + r < N)
        {
          const T x = FAST ? v[(r0 + r) * N + j] : v[j * N + r0 + r];
#pragma unroll
          for (int i = 0; i < N; i++)
            w[r][i] = fma(a[i], x, j ? w[r][i] : T(0));
        }
    }
#pragma unroll
    for (int r = 0; r < RB; r++)
      if (r0 + r < N)
#pragma unroll
        for (int i = 0; i < N; i++)
          v[FAST ? (r0 + r) * N + i : i * N + r0 + r] = w[r][i];
  }
}

template <typename T, int D, int N, bool MERGE>
__global__ void __launch_bounds__(PairShape<T, D, N, MERGE>::THREADS)
    kron_pair_kernel(const __grid_constant__ Params p)
{
  using S = PairShape<T, D, N, MERGE>;
  constexpr int L = S::L, N2 = S::N2, F = S::F, CS = S::CS, GS = S::THREADS, V = S::V;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ const T *s_ptr[3][8]; // A_1..A_d, x at 6, y at 7, of three entries
  const int t = threadIdx.x;
  int e, ee;
  group_range(p, blockIdx.x, gridDim.x, e, ee);
  if (e >= ee)
    return;
  T *stage0 = reinterpret_cast<T *>(smem);
  T *sum    = stage0 + S::STAGES * S::XLEN; // MERGE
  T *fac0   = stage0 + (S::STAGES + (MERGE ? 1 : 0)) * S::XLEN;

  const bool a_ptrs = p.layout != LAYOUT_BATCHED && p.layout != LAYOUT_PBATCHED;
  const bool x_ptrs = p.layout != LAYOUT_BATCHED;
  const int ld      = p.layout == LAYOUT_XBATCHED ? p.lda : N;
  auto pointer = [&](int e, int j) -> const T * {
    const int k = entry_index(p, e);
    if (j < D)
      return a_ptrs ? static_cast<const T *>(p.pA[(long long)k * p.apk + j])
                    : static_cast<const T *>(p.A) + ((long long)k * D + j) * N2;
    if (j == 6)
      return x_ptrs ? static_cast<const T *>(p.pX[k])
                    : static_cast<const T *>(p.X) + (long long)k * p.xstride;
    if (j == 7)
      return x_ptrs ? static_cast<const T *>(p.pY[k])
                    : static_cast<const T *>(p.Y) + (long long)k * p.ystride;
    return nullptr;
  };
  // x of an entry into a stage, its factors into set b
  auto issue = [&](const T *const *ptr, T *st, int b) {
    const T *x = ptr[6];
    if (S::VEC && aligned16(x))
    {
      for (int u = t; u < L / V; u += GS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(st + S::pos(u * V))),
                     "l"(x + u * V)
                     : "memory");
    }
    else
      for (int u = t; u < L; u += GS)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(st + S::pos(u))),
                     "l"(x + u), "n"((int)sizeof(T))
                     : "memory");
    T *as = fac0 + b * D * S::AF;
    for (int q = t; q < D * N2; q += GS)
    {
      const int l = q / N2, j = (q - l * N2) / N, i = q - l * N2 - j * N;
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(as + l * S::AF + j * S::LD + i)),
                   "l"(ptr[l] + i + (long long)j * ld), "n"((int)sizeof(T))
                   : "memory");
    }
  };

  if (t < 8)
  {
    s_ptr[0][t] = pointer(e, t);
    if (e + 1 < ee)
      s_ptr[1][t] = pointer(e + 1, t);
  }
  __syncthreads();
  issue(s_ptr[0], stage0, 0);
  bool have = false; // MERGE: sum holds results of this run of equal outputs
  for (int i = 0;; i++)
  {
    const int b     = i & 1;
    const bool more = e + 1 < ee;
    T *st           = stage0 + (S::STAGES == 2 ? b * S::XLEN : 0);
    const T *as     = fac0 + b * D * S::AF;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const T *const *next = s_ptr[(i + 1) % 3];
    const T *far         = nullptr;
    if (more)
    {
      if constexpr (S::STAGES == 2)
        issue(next, stage0 + (b ^ 1) * S::XLEN, b ^ 1);
      else
        for (int q = t; q < L * (int)sizeof(T) / 128; q += GS)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next[6] + q * (128 / (int)sizeof(T))));
      if (t < 8 && e + 2 < ee)
        far = pointer(e + 2, t);
    }
    T *y = const_cast<T *>(s_ptr[i % 3][7]);

    // ---- modes 1, 2: elements c n^(d-2) + f
    for (int f = t; f < F; f += GS)
    {
      constexpr int ST = F / N2 * CS; // a step of mode 2 (F is a multiple of n^2)
      T *x = st + f / N2 * CS + f % N2;
      T v[N2];
#pragma unroll
      for (int c = 0; c < N2; c++)
        v[c] = x[c * ST];
      pair_apply<T, N, S::LD, S::RB, false>(v, as);
      pair_apply<T, N, S::LD, S::RB, true>(v, as + S::AF);
#pragma unroll
      for (int c = 0; c < N2; c++)
        x[c * ST] = v[c];
    }
    __syncthreads();
    // ---- d = 5, 6: modes 3, 4 with n or n^2 elements of the later modes inside
    if constexpr (D > 4)
    {
      constexpr int IN = D == 5 ? N : N2;
      for (int f = t; f < F; f += GS)
      {
        const int o = f / IN, r = f - o * IN;
        T *x = st + o * (IN * CS) + r;
        T v[N2];
#pragma unroll
        for (int c = 0; c < N2; c++)
          v[c] = x[c * IN / N2 * CS + c * IN % N2];
        pair_apply<T, N, S::LD, S::RB, false>(v, as + 2 * S::AF);
        pair_apply<T, N, S::LD, S::RB, true>(v, as + 3 * S::AF);
#pragma unroll
        for (int c = 0; c < N2; c++)
          x[c * IN / N2 * CS + c * IN % N2] = v[c];
      }
      __syncthreads();
    }
    // ---- the last two modes (d = 5: the last) on contiguous fibres
    for (int f = t; f < F; f += GS)
    {
      T v[N2];
      load_chunk<T, N>(st + f * CS, v);
      if constexpr (D != 5)
        pair_apply<T, N, S::LD, S::RB, false>(v, as + (D - 2) * S::AF);
      pair_apply<T, N, S::LD, S::RB, true>(v, as + (D - 1) * S::AF);
      if constexpr (MERGE)
      {
        if (have)
        {
#pragma unroll
          for (int c0 = 0; c0 < N2; c0 += N)
          {
            T o[N];
#pragma unroll
            for (int c = 0; c < N; c++)
              o[c] = sum[f * CS + c0 + c];
#pragma unroll
            for (int c = 0; c < N; c++)
              v[c0 + c] += o[c];
          }
        }
        store_chunk<T, N>(sum + f * CS, v);
      }
      else
        store_chunk<T, N>(st + f * CS, v);
    }
    // ---- results
    have = MERGE && more && next[7] == y;
    if (!have)
    {
      const T *res = MERGE ? sum : st;
      __syncthreads();
      if constexpr (sizeof(T) == 8)
      {
#pragma unroll 4
        for (int q = t; q < L; q += GS)
          red_add(y + q, res[S::pos(q)]);
      }
      else
      {
        for (int q0 = t; q0 < L; q0 += 8 * GS)
        {
          T old[8];
#pragma unroll
          for (int c = 0; c < 8; c++)
            if (q0 + c * GS < L)
              old[c] = y[q0 + c * GS];
#pragma unroll
          for (int c = 0; c < 8; c++)
            if (q0 + c * GS < L)
              y[q0 + c * GS] = old[c] + res[S::pos(q0 + c * GS)];
        }
      }
    }
    if (!more)
      break;
    if constexpr (S::STAGES == 1)
    {
      __syncthreads();
      issue(next, stage0, b ^ 1);
    }
    if (t < 8 && e + 2 < ee)
      s_ptr[(i + 2) % 3][t] = far;
    ++e;
  }
}

template <typename T, int D, int N, bool MERGE>
int launch_pair_t(Params p, cudaStream_t stream)
{
  using S        = PairShape<T, D, N, MERGE>;
  const void *fn = reinterpret_cast<const void *>(&kron_pair_kernel<T, D, N, MERGE>);
  int per_sm     = 1;
  if (cached_occupancy(fn, S::THREADS, S::SMEM, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  const long long work = p.seg_off ? p.nitems : (long long)p.eend - p.ebase;
  const long long grid = std::min<long long>(work, (long long)device_info().sms * per_sm);
  void *args[]         = {&p};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(S::THREADS), args, S::SMEM, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

// the form with sums in shared memory where outputs may repeat and it fits
template <typename T, int D, int N>
int launch_pair_m(const Params &p, cudaStream_t stream)
{
  if constexpr (sizeof(T) == 8 && PairShape<T, D, N, true>::SMEM <= 224 * 1024)
    if (p.accum != ACC_DISTINCT)
      return launch_pair_t<T, D, N, true>(p, stream);
  // a segment is one add an element
  return p.seg_off ? KRON_ERROR_NOT_SUPPORTED : launch_pair_t<T, D, N, false>(p, stream);
}

template <typename T>
int pair_pick(const Params &p, cudaStream_t s)
{
  switch (p.n[0] * 8 + p.d)
  {
  case 3 * 8 + 6: return launch_pair_m<T, 6, 3>(p, s);
  case 4 * 8 + 5: return launch_pair_m<T, 5, 4>(p, s);
  case 5 * 8 + 4: return launch_pair_m<T, 4, 5>(p, s);
  case 5 * 8 + 5: return launch_pair_m<T, 5, 5>(p, s);
  case 5 * 8 + 6: return launch_pair_m<T, 6, 5>(p, s);
  case 6 * 8 + 4: return launch_pair_m<T, 4, 6>(p, s);
  case 6 * 8 + 5: return launch_pair_m<T, 5, 6>(p, s);
  case 7 * 8 + 4: return launch_pair_m<T, 4, 7>(p, s);
  case 7 * 8 + 5: return launch_pair_m<T, 5, 7>(p, s);
  case 8 * 8 + 4: return launch_pair_m<T, 4, 8>(p, s);
  default: return KRON_ERROR_NOT_SUPPORTED;
  }
}

} // namespace

bool pair_supported(const Params &p, int prec)
{
  // FP32 outputs are exclusive (there is only the batched layout)
  if (p.accum == ACC_STORE || !(prec == PREC_F64 || (prec == PREC_F32 && p.accum == ACC_DISTINCT)))
    return false;
  for (int l = 0; l < p.d; l++)
    if (p.m[l] != p.n[0] || p.n[l] != p.n[0])
      return false;
  return true;
}

int launch_pair(const Params &p, int prec, cudaStream_t stream)
{
  if (p.eend <= p.ebase)
    return KRON_SUCCESS;
  return prec == PREC_F32 ? pair_pick<float>(p, stream) : pair_pick<double>(p, stream);
}

} // namespace kron
