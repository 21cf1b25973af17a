// Register-blocked fibres of two modes: an n x n block of a vector held by one
// thread, v[a n + b], with b the faster mode, and the products of it with one
// n x n factor along either mode.  Shared by the slab-cluster, resident, ring
// and pair kernels.
#pragma once

#include <type_traits>

#include "kron_internal.cuh"

namespace kron {

// factor A (column major, A(i, j) at i + j N) into registers
template <typename T, int N>
__device__ __forceinline__ void load_factor(const T *A, T (&a)[N][N])
{
#pragma unroll
  for (int j = 0; j < N; j++)
  {
    if constexpr (sizeof(T) == 8 && N % 2 == 0)
    {
#pragma unroll
      for (int i = 0; i < N; i += 2)
      {
        const double2 u = *reinterpret_cast<const double2 *>(A + i + j * N);
        a[i][j]         = u.x;
        a[i + 1][j]     = u.y;
      }
    }
    else if constexpr (sizeof(T) == 4 && N % 2 == 0)
    {
#pragma unroll
      for (int i = 0; i < N; i += 2)
      {
        const float2 u = *reinterpret_cast<const float2 *>(A + i + j * N);
        a[i][j]        = u.x;
        a[i + 1][j]    = u.y;
      }
    }
    else
    {
#pragma unroll
      for (int i = 0; i < N; i++)
        a[i][j] = A[i + j * N];
    }
  }
}

// v is an n x n block, v[a N + b]: apply_fast applies A along b (the faster
// mode), apply_slow along a
template <typename T, int N>
__device__ __forceinline__ void apply_fast(T (&v)[N * N], const T *A)
{
  T a[N][N];
  load_factor<T, N>(A, a);
#pragma unroll
  for (int r = 0; r < N; r++)
  {
    T t[N];
#pragma unroll
    for (int i = 0; i < N; i++)
    {
      T z = a[i][0] * v[r * N];
#pragma unroll
      for (int j = 1; j < N; j++)
        z = fma(a[i][j], v[r * N + j], z);
      t[i] = z;
    }
#pragma unroll
    for (int i = 0; i < N; i++)
      v[r * N + i] = t[i];
  }
}

template <typename T, int N>
__device__ __forceinline__ void apply_slow(T (&v)[N * N], const T *A, int rot = 0)
{
  T a[N][N];
  if (rot == 0)
    load_factor<T, N>(A, a);
  else
  {
    // rows of v hold rows (r + rot) mod N: the factor with rows and columns
    // rotated the same way gives the rotated rows of the product
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++)
      {
        const int ri = i + rot < N ? i + rot : i + rot - N;
        const int rj = j + rot < N ? j + rot : j + rot - N;
        a[i][j]      = A[ri + rj * N];
      }
  }
#pragma unroll
  for (int c = 0; c < N; c++)
  {
    T t[N];
#pragma unroll
    for (int i = 0; i < N; i++)
    {
      T z = a[i][0] * v[c];
#pragma unroll
      for (int j = 1; j < N; j++)
        z = fma(a[i][j], v[j * N + c], z);
      t[i] = z;
    }
#pragma unroll
    for (int i = 0; i < N; i++)
      v[i * N + c] = t[i];
  }
}

// A contiguous fibre from / to shared memory, 16 bytes at a time when n is even
// (b 16-byte aligned).
template <typename T, int N>
__device__ __forceinline__ void load_chunk(const T *b, T (&v)[N * N])
{
  if constexpr (N % 2 == 0)
  {
    constexpr int V = 16 / sizeof(T);
    using VT        = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
#pragma unroll
    for (int c = 0; c < N * N; c += V)
    {
      const VT u = *reinterpret_cast<const VT *>(b + c);
      v[c]       = u.x;
      v[c + 1]   = u.y;
      if constexpr (V == 4)
      {
        v[c + 2] = u.z;
        v[c + 3] = u.w;
      }
    }
  }
  else
  {
#pragma unroll
    for (int c = 0; c < N * N; c++)
      v[c] = b[c];
  }
}

template <typename T, int N>
__device__ __forceinline__ void store_chunk(T *b, const T (&v)[N * N])
{
  if constexpr (N % 2 == 0 && sizeof(T) == 8)
  {
#pragma unroll
    for (int c = 0; c < N * N; c += 2)
      *reinterpret_cast<double2 *>(b + c) = make_double2(v[c], v[c + 1]);
  }
  else if constexpr (N % 2 == 0)
  {
#pragma unroll
    for (int c = 0; c < N * N; c += 4)
      *reinterpret_cast<float4 *>(b + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
  }
  else
  {
#pragma unroll
    for (int c = 0; c < N * N; c++)
      b[c] = v[c];
  }
}

} // namespace kron
