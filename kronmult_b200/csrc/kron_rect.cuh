// Mode products of runtime (rectangular) shapes, prepared on the host.
//
// A vector's mode products run as a list of steps, each out of place on
// fibres of one mode: fibre f = (o, r), o = f / inner, reads
// cur[(o nq + j) inner + r] and writes nxt[(o mq + i) inner + r].  The list
// is computed once (per launch or per plan), so that a thread's work per step
// is its fibres only: no shapes to multiply out, and o by a multiplication.
// The factors lie in shared memory in the order of the steps.
#pragma once

#include <cmath>

#include "kron_internal.cuh"

namespace kron {

struct RectStep
{
  int inner;          // elements between consecutive indices of the mode
  int nfib;           // fibres (of one row, where the buffer holds several)
  unsigned magic;     // ceil(2^32 / inner), 0 for inner = 1
  unsigned char nq, mq, mode, pad;
};
static_assert(sizeof(RectStep) == 16, "read as one 16-byte word");

// Steps of the modes [mode0, mode0 + dd) in the given order; C columns ride
// along as the fastest index.  Exact while the elements of a buffer times the
// largest inner stay below 2^32 (buffers fit shared memory).
inline void rect_plan(RectStep *st, int dd, const int *m, const int *n, int mode0, bool forward,
                      int C)
{
  // `left`: the modes not yet applied (their input sizes), `done`: the applied
  // ones (their output sizes), with the columns on the fastest side
  unsigned left[MAXD + 1], done = forward ? 1u : (unsigned)C;
  left[dd] = 1;
  for (int s = dd - 1; s >= 0; s--)
    left[s] = left[s + 1] * (unsigned)n[forward ? s : dd - 1 - s];
  for (int s = 0; s < dd; s++)
  {
    const int q          = forward ? s : dd - 1 - s;
    const unsigned inner = forward ? left[s + 1] * (unsigned)C : done;
    st[s].inner = (int)inner;
    st[s].nfib  = (int)(forward ? done * inner : left[s + 1] * inner);
    // exact in double: the quotient has 32 bits, its fraction at least 1 / inner
    st[s].magic = inner == 1 ? 0u : (unsigned)std::ceil(4294967296.0 / inner);
    st[s].nq    = (unsigned char)n[q];
    st[s].mq    = (unsigned char)m[q];
    st[s].mode  = (unsigned char)(mode0 + q);
    st[s].pad   = 0;
    done *= (unsigned)m[q];
  }
}

// Factors of up to AREG_MAX elements are held in registers, larger ones are read
// from shared memory at every use.
template <typename T, int AREG_MAX, int NQ, int MQ>
__device__ __forceinline__ void rect_fibres(const T *cur, T *nxt, const T *A, int inner,
                                            unsigned magic, int nfib, int t, int GS)
{
  constexpr bool AREG = NQ * MQ <= AREG_MAX;
  T a[AREG ? MQ : 1][AREG ? NQ : 1];
  if constexpr (AREG)
  {
    if (t < nfib)
#pragma unroll
      for (int j = 0; j < NQ; j++)
#pragma unroll
        for (int i = 0; i < MQ; i++)
          a[i][j] = A[i + j * MQ];
  }
  for (int f = t; f < nfib; f += GS)
  {
    const int o  = magic ? (int)__umulhi((unsigned)f, magic) : f;
    const int oi = o * inner;
    const T *src = cur + f + oi * (NQ - 1);
    T *dst       = nxt + f + oi * (MQ - 1);
    T x[NQ];
#pragma unroll
    for (int j = 0; j < NQ; j++)
      x[j] = src[j * inner];
#pragma unroll
    for (int i = 0; i < MQ; i++)
    {
      T z = T(0);
#pragma unroll
      for (int j = 0; j < NQ; j++)
        z = fma(AREG ? a[AREG ? i : 0][AREG ? j : 0] : A[i + j * MQ], x[j], z);
      dst[i * inner] = z;
    }
  }
}

// The innermost mode (inner = 1), a thread an output element: fibres a thread
// apart would be read at a stride of NQ elements and written at one of MQ, up to
// eight bank passes an access.  Here the threads of a fibre read the same element
// and writes are contiguous; a thread keeps its row of the factor, NQ elements.
// (Threads beyond a whole number of fibres have no work.)  4096 entries of 576
// elements: 32.8 -> 30.5 us; uneven plans, whose items hold many more fibres,
// lose 0.4% and keep the fibres.
template <typename T, int NQ, int MQ>
__device__ __forceinline__ void rect_innermost(const T *cur, T *nxt, const T *A, int nfib, int t,
                                               int GS)
{
  const int per = GS / MQ; // fibres a round
  const int o0 = t / MQ, i = t - o0 * MQ;
  if (o0 >= per || o0 >= nfib)
    return;
  T a[NQ];
#pragma unroll
  for (int j = 0; j < NQ; j++)
    a[j] = A[i + j * MQ];
  for (int o = o0; o < nfib; o += per)
  {
    const T *src = cur + o * NQ;
    T z          = T(0);
#pragma unroll
    for (int j = 0; j < NQ; j++)
      z = fma(a[j], src[j], z);
    nxt[o * MQ + i] = z;
  }
}

// Sizes beyond 8: a thread an output element, so that short vectors with long
// modes keep the whole group at work (a thread a fibre left one thread of 32 for
// d = 1, n = 64, 32 of 128 for d = 2, n = 32: 100 entries 53 -> 12 and 95 -> 12
// us, the larger groups of kron_rect.cu included).  Neighbouring threads read
// neighbouring elements of x or of a column of the factor, and the same of the other.
template <typename T>
__device__ __noinline__ void rect_step_any(const T *cur, T *nxt, const T *A, int nq, int mq,
                                           int inner, unsigned magic, int nfib, int t, int GS)
{
  const int total = nfib * mq;
  for (int f = t; f < total; f += GS)
  {
    // f = (o mq + i) inner + r
    const int oi = magic ? (int)__umulhi((unsigned)f, magic) : f, r = f - oi * inner;
    const int o  = oi / mq, i = oi - o * mq;
    const T *src = cur + o * nq * inner + r, *a = A + i;
    T z          = T(0);
#pragma unroll 4
    for (int j = 0; j < nq; j++)
      z = fma(a[j * mq], src[j * inner], z);
    nxt[f] = z;
  }
}

// all steps over `rows` consecutive vectors; cur holds the result at the end
template <typename T, int AREG_MAX, bool BY_OUTPUT = false>
__device__ __forceinline__ void rect_modes(const RectStep *st, int ns, int rows, T *&cur, T *&nxt,
                                           const T *As, int t, int GS, int g)
{
  for (int s = 0; s < ns; s++)
  {
    const RectStep q = st[s];
    const int nfib   = q.nfib * rows, inner = q.inner;
    switch (q.nq <= 8 && q.mq <= 8 ? q.nq * 16 + q.mq : 0)
    {
#define KRON_RM(NQ_, MQ_)                                                                       \
  case NQ_ * 16 + MQ_:                                                                          \
    if (BY_OUTPUT && MQ_ > 1 && inner == 1)                                                     \
      rect_innermost<T, NQ_, MQ_>(cur, nxt, As, nfib, t, GS);                                   \
    else                                                                                        \
      rect_fibres<T, AREG_MAX, NQ_, MQ_>(cur, nxt, As, inner, q.magic, nfib, t, GS);            \
    break;
#define KRON_RM_ROW(NQ_)                                                                        \
  KRON_RM(NQ_, 1) KRON_RM(NQ_, 2) KRON_RM(NQ_, 3) KRON_RM(NQ_, 4) KRON_RM(NQ_, 5)              \
  KRON_RM(NQ_, 6) KRON_RM(NQ_, 7) KRON_RM(NQ_, 8)
      KRON_RM_ROW(1) KRON_RM_ROW(2) KRON_RM_ROW(3) KRON_RM_ROW(4)
      KRON_RM_ROW(5) KRON_RM_ROW(6) KRON_RM_ROW(7) KRON_RM_ROW(8)
#undef KRON_RM_ROW
#undef KRON_RM
    default: rect_step_any(cur, nxt, As, q.nq, q.mq, inner, q.magic, nfib, t, GS); break;
    }
    As += q.nq * q.mq;
    T *tmp = cur;
    cur    = nxt;
    nxt    = tmp;
    group_sync(g, GS);
  }
}

} // namespace kron
