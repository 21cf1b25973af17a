// Packed kernel: short vectors of low-order elements (square n = 2..5, d >= 3,
// at most 32 fibres of n^2 elements), FP64 and FP32, every layout and
// accumulation mode.
//
// These calls are bound inside the SM, not by bytes or flops: the square
// kernel issued 365 warp instructions for an entry of 81 elements (d = 4, n =
// 3), this one 239, and the data pipe of shared memory, 111 passes an entry, is
// 81% busy while its warps run.  Here a warp computes up to four entries at a time, a lane a fibre of
// two modes in registers: half the passes, and each instruction serves
// several entries.  A warp works through a contiguous, balanced range of
// entries with the next ones' factors and vectors on their way to shared
// memory (cp.async, two stages) and the pointers of those after next on
// their way to registers (lane 8 s + j holds pointer j of the warp's entry s).
// Warps share nothing; all barriers are the warp's.  36000 entries with shared
// factors, 4000 outputs, FP64, packed against square kernel: d = 4, n = 3 20.7
// against 26.9 us; d = 4, n = 4 31 against 78; d = 6, n = 2 16.6 against 24.8;
// d = 5, n = 3 43 against 64 (49 with four blocks a multiprocessor: 64
// registers spill).
//
// Results of consecutive entries with the same output are summed in registers
// and added into y once, by red.global.add: with exclusive or segmented
// outputs each element gets exactly one add a call, so sums are bitwise
// reproducible.  FP32 (exclusive outputs only) loads y ahead of the products and
// stores the sum: an FP32 add in the L2 cache would flush subnormals.
//
// (The reference runs one 64-thread block per entry through global memory,
// kronmult_xbatched.hpp:17-162.)
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kron_launch.h"
#include "kron_ptx.cuh"

namespace kron {

namespace {

using namespace ptx;

constexpr int PACK_WARPS = 8;

template <typename T, int D, int N>
struct PackShape
{
  static constexpr int N2  = N * N;
  static constexpr int L   = cpow(N, D);
  static constexpr int F   = L / N2; // fibres of two modes
  static constexpr int EPW = F > 16 ? 1 : (F > 10 ? 2 : (F > 8 ? 3 : 4)); // entries a warp
  static constexpr int ASZ = D * N2;
  static_assert(F * EPW <= 32, "a fibre a lane");
  // for even n one element of padding after every 16: lanes n^2 elements apart
  // do not meet in the same banks (odd n: n^2 is odd)
  static constexpr bool PAD = N % 2 == 0;
  static constexpr int V    = 16 / (int)sizeof(T);
  static constexpr int XLEN = ((PAD ? L + (L - 1) / 16 : L) + V - 1) / V * V;
  // a factor starts on a 16-byte boundary, so that it is read 16 bytes at a time
  static constexpr int AF   = (N2 + V - 1) / V * V;
  static constexpr int SLOT = XLEN + D * AF; // elements of an entry in a stage
  static constexpr int STAGE = (EPW * SLOT + 3) / 4 * 4;
  static constexpr int PER  = (L + 31) / 32; // elements of y a lane
  __device__ static __forceinline__ constexpr int pos(int i) { return PAD ? i + i / 16 : i; }
};

template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src),
               "n"((int)sizeof(T))
               : "memory");
}

// Modes [a, a + k) (k = 1, 2) of the entry at x, lane's fibre f of its n^d / n^k.
template <typename T, int D, int N, int a, int k>
__device__ __forceinline__ void pack_pass(T *x, const T *A, int f)
{
  using S         = PackShape<T, D, N>;
  constexpr int ST = cpow(N, D - a - k); // stride of the last of the modes
  constexpr int C  = cpow(N, k);
  const int o = f / ST, r = f - o * ST, base = o * (C * ST) + r;
  T v[C];
#pragma unroll
  for (int c = 0; c < C; c++)
    v[c] = x[S::pos(base + c * ST)];
#pragma unroll
  for (int m = 0; m < k; m++) // in the square kernel's order: the same products, bit for bit
  {
    T A_[S::AF]; // the factor, column major
#pragma unroll
    for (int u = 0; u < S::AF; u += S::V)
    {
      using VT   = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
      const VT q = *reinterpret_cast<const VT *>(A + (a + m) * S::AF + u);
      A_[u]      = q.x;
      A_[u + 1]  = q.y;
      if constexpr (S::V == 4)
      {
        A_[u + 2] = q.z;
        A_[u + 3] = q.w;
      }
    }
    T w[C];
#pragma unroll
    for (int c = 0; c < C; c++)
      w[c] = T(0);
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int i = 0; i < N; i++)
      {
        const T c = A_[i + j * N];
        // fibres of mode a + m inside the fibre
#pragma unroll
        for (int q = 0; q < C / N; q++)
        {
          const int b = (m == k - 1) ? q * N : q; // fast mode: rows; slow: columns
          const int s = (m == k - 1) ? 1 : N;
          w[b + i * s] = fma(c, v[b + j * s], w[b + i * s]);
        }
      }
#pragma unroll
    for (int c = 0; c < C; c++)
      v[c] = w[c];
  }
#pragma unroll
  for (int c = 0; c < C; c++)
    x[S::pos(base + c * ST)] = v[c];
}

template <typename T, int D, int N, int a = 0>
__device__ __forceinline__ void pack_passes(T *x, const T *A, int f, bool on)
{
  using S = PackShape<T, D, N>;
  if constexpr (a + 2 <= D)
  {
    if (on)
      pack_pass<T, D, N, a, 2>(x, A, f);
    __syncwarp();
    pack_passes<T, D, N, a + 2>(x, A, f, on);
  }
  else if constexpr (a + 1 == D)
  {
    // the odd mode: n times the fibres, of n elements
    if (on)
#pragma unroll
      for (int q = 0; q < N; q++)
        pack_pass<T, D, N, a, 1>(x, A, f + q * S::F);
    __syncwarp();
  }
}

template <typename T, int D, int N>
__global__ void __launch_bounds__(PACK_WARPS * 32, N > 3 ? 2 : (N == 3 && D == 5 ? 3 : 4))
    kron_pack_kernel(const __grid_constant__ Params p)
{
  using S           = PackShape<T, D, N>;
  constexpr int L = S::L, N2 = S::N2, EPW = S::EPW, ASZ = S::ASZ;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T *base        = reinterpret_cast<T *>(smem) + warp * 2 * S::STAGE;
  int e, ee;
  group_range(p, blockIdx.x * PACK_WARPS + warp, gridDim.x * PACK_WARPS, e, ee);
  if (e >= ee)
    return;

  const bool a_ptrs = p.layout != LAYOUT_BATCHED && p.layout != LAYOUT_PBATCHED;
  const bool x_ptrs = p.layout != LAYOUT_BATCHED;
  const int ld      = p.layout == LAYOUT_XBATCHED ? p.lda : N;
  // lane 8 s + j: pointer j (A_1..A_d at 0.., x at 6, y at 7) of position e + s
  auto pointers = [&](int e) -> const T * {
    const int s = lane >> 3, j = lane & 7;
    if (s >= EPW || e + s >= ee)
      return nullptr;
    const int k = entry_index(p, e + s);
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
  auto of_lane = [&](const T *ptr, int l) {
    return reinterpret_cast<const T *>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(ptr), l));
  };
  // factors and vectors of the entries whose pointers the lanes hold (those
  // past the range have none)
  auto issue = [&](const T *ptr, T *st, int count) {
#pragma unroll
    for (int s = 0; s < EPW; s++)
      if (s < count)
      {
        T *xs = st + s * S::SLOT, *as = xs + S::XLEN;
        const T *x = of_lane(ptr, 8 * s + 6);
#pragma unroll
        for (int i0 = 0; i0 < L; i0 += 32)
          if (L % 32 == 0 || i0 + lane < L)
            cp_async_elem(xs + S::pos(i0 + lane), x + i0 + lane);
        if (!a_ptrs)
        {
          const T *A = of_lane(ptr, 8 * s); // A_1..A_d contiguous
#pragma unroll
          for (int q0 = 0; q0 < ASZ; q0 += 32)
            if (ASZ % 32 == 0 || q0 + lane < ASZ)
              cp_async_elem(as + q0 + lane + (S::AF - N2) * ((q0 + lane) / N2), A + q0 + lane);
        }
        else
#pragma unroll
          for (int q0 = 0; q0 < ASZ; q0 += 32)
          {
            const int q = q0 + lane, l = min(q / N2, D - 1), ij = q - l * N2, j = ij / N;
            const T *A  = of_lane(ptr, 8 * s + l);
            if (ASZ % 32 == 0 || q < ASZ)
              cp_async_elem(as + l * S::AF + ij, A + (ij - j * N) + j * ld);
          }
      }
  };

  // this lane's entry of the warp's and fibre
  const int slot = min(lane / S::F, EPW - 1), f = lane - slot * S::F;
  const bool mine = f < S::F;
  const T *pc = pointers(e), *pn = nullptr;
  issue(pc, base, min(EPW, ee - e));
  if (e + EPW < ee)
    pn = pointers(e + EPW);
  T acc[S::PER];
#pragma unroll
  for (int j = 0; j < S::PER; j++)
    acc[j] = T(0);

  for (int b = 0;; b ^= 1)
  {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    T *st           = base + b * S::STAGE;
    const int count = min(EPW, ee - e);
    const bool more = e + EPW < ee;
    const T *py     = pc;
    if (more)
    {
      issue(pn, base + (b ^ 1) * S::STAGE, min(EPW, ee - e - EPW));
      pc = pn;
      if (e + 2 * EPW < ee)
        pn = pointers(e + 2 * EPW);
    }
    // FP32: y is on its way during the products
    T old[sizeof(T) == 4 ? EPW : 1][S::PER];
    if constexpr (sizeof(T) == 4)
#pragma unroll
      for (int s = 0; s < EPW; s++)
        if (s < count)
        {
          const T *ys = of_lane(py, 8 * s + 7);
#pragma unroll
          for (int j = 0; j < S::PER; j++)
            if (L % 32 == 0 || lane + 32 * j < L)
              old[s][j] = ys[lane + 32 * j];
        }
    T *xs = st + slot * S::SLOT;
    pack_passes<T, D, N>(xs, xs + S::XLEN, f, mine && slot < count);
    // outputs, entry by entry; the sum goes out where the output changes
    T *y = const_cast<T *>(of_lane(py, 7));
#pragma unroll
    for (int s = 0; s < EPW; s++)
      if (s < count)
      {
        // the next entry's output (of the next step after the last)
        const T *yn;
        if (s + 1 < EPW)
          yn = of_lane(py, min(8 * (s + 1) + 7, 31));
        else
          yn = of_lane(pc, 7);
        const bool last = s + 1 < count ? false : !more;
        const T *vs     = st + s * S::SLOT;
#pragma unroll
        for (int j = 0; j < S::PER; j++)
          if (L % 32 == 0 || lane + 32 * j < L)
          {
            if constexpr (sizeof(T) == 4)
              y[lane + 32 * j] = old[s][j] + vs[S::pos(lane + 32 * j)];
            else
              acc[j] += vs[S::pos(lane + 32 * j)];
          }
        if constexpr (sizeof(T) == 8)
          if (last || yn != y)
          {
#pragma unroll
            for (int j = 0; j < S::PER; j++)
            {
              if (L % 32 == 0 || lane + 32 * j < L)
                red_add(y + lane + 32 * j, acc[j]);
              acc[j] = T(0);
            }
          }
        y = const_cast<T *>(yn);
      }
    if (!more)
      break;
    e += EPW;
    __syncwarp(); // every lane has read the stage that the next copies overwrite
  }
}

template <typename T, int D, int N>
int launch_pack_t(Params p, cudaStream_t stream)
{
  using S           = PackShape<T, D, N>;
  const void *fn    = reinterpret_cast<const void *>(&kron_pack_kernel<T, D, N>);
  const size_t smem = PACK_WARPS * 2 * (size_t)S::STAGE * sizeof(T);
  int per_sm        = 1;
  if (cached_occupancy(fn, PACK_WARPS * 32, smem, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  const long long work = p.seg_off ? p.nitems : (long long)p.eend - p.ebase;
  const long long grid = std::min<long long>((work + PACK_WARPS - 1) / PACK_WARPS,
                                             (long long)device_info().sms * per_sm);
  void *args[] = {&p};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(PACK_WARPS * 32), args, smem, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

template <typename T>
int pack_pick(const Params &p, cudaStream_t s)
{
  switch (p.n[0] * 8 + p.d)
  {
  case 2 * 8 + 3: return launch_pack_t<T, 3, 2>(p, s);
  case 2 * 8 + 4: return launch_pack_t<T, 4, 2>(p, s);
  case 2 * 8 + 5: return launch_pack_t<T, 5, 2>(p, s);
  case 2 * 8 + 6: return launch_pack_t<T, 6, 2>(p, s);
  case 3 * 8 + 3: return launch_pack_t<T, 3, 3>(p, s);
  case 3 * 8 + 4: return launch_pack_t<T, 4, 3>(p, s);
  case 3 * 8 + 5: return launch_pack_t<T, 5, 3>(p, s);
  case 4 * 8 + 3: return launch_pack_t<T, 3, 4>(p, s);
  case 4 * 8 + 4: return launch_pack_t<T, 4, 4>(p, s);
  case 5 * 8 + 3: return launch_pack_t<T, 3, 5>(p, s);
  default: return KRON_ERROR_NOT_SUPPORTED;
  }
}

} // namespace

bool pack_supported(const Params &p, int prec)
{
  // FP32 outputs are exclusive (there is only the batched layout)
  if (p.accum == ACC_STORE || !(prec == PREC_F64 || (prec == PREC_F32 && p.accum == ACC_DISTINCT)))
    return false;
  const int n = p.n[0];
  for (int l = 0; l < p.d; l++)
    if (p.m[l] != n || p.n[l] != n)
      return false;
  if (p.d < 3)
    return false;
  return n == 2 || (n == 3 && p.d <= 5) || (n == 4 && p.d <= 4) || (n == 5 && p.d == 3);
}

int launch_pack(const Params &p, int prec, cudaStream_t stream)
{
  if (p.eend <= p.ebase)
    return KRON_SUCCESS;
  return prec == PREC_F32 ? pack_pick<float>(p, stream) : pack_pick<double>(p, stream);
}

} // namespace kron
