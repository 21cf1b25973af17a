// Ring kernel: square d = 6 vectors beyond one block's shared memory (n = 6..8,
// FP64 and FP32: 187 KB .. 2 MB per entry), with a workspace W.
//
// The six modes split into a head (slow) and a tail (fast) group, x viewed as
// LH head rows of LT contiguous elements:
//   phase 1: a few head rows at a time get the tail modes; results -> W;
//   phase 2: a few columns of W at a time get the head modes; results are
//            added into y by red.global.add.
// (The recursive algorithm's two-level split, kronmultv_recur.hpp:117-145.)
//
// Every entry is cut into K equal parts of each phase.  One queue orders all
// parts: item g K + r is part r of entry g's phase 1 and part r of entry
// (g - lag)'s phase 2.  Blocks take items in order from a device counter, so
// an item waits only for items that running blocks already hold: phase 2 for
// its entry's K phase-1 parts, lag groups back (normally long done), and
// phase 1 for the ring slot of W it writes, last read by the entry `slots`
// positions back.  W is a ring of `slots` vectors, a few tens of MB that stay
// in the L2 cache however large the batch; no cluster barriers, and every SM
// works on both phases, so loads of x, math and adds into y overlap between
// the blocks of an SM.
//
// The control words (queue, abort, and per slot the parts done of each phase,
// counted up over the slot's generations) lie in the workspace vector after
// the ring, zeroed by a small kernel ahead of this one.  A block publishes an
// item's parts in the middle of the next item, when its stores have long
// drained (a fence behind fresh stores and adds takes 2-3 us here), with one
// fence for both counters and for the look at the next item's dependencies.  Waits are bounded (wait_limit() polls): a block that
// gives up records 1 in the device status word, raises the abort word, which
// ends the others' waits, and leaves; y of the parts not done is untouched.
//
// Measured against what ran before (the cluster two-phase kernel, whose W
// goes through HBM and back: 9.35 against 6.9 GB for 1024 entries of n = 8;
// n = 6: the slab-cluster kernel with its side kernel):
//   n = 6, 4096 entries  1.397 -> 1.289 ms (HBM alone 0.70)
//   n = 7, 256 entries   0.465 -> 0.256 ms (HBM alone 0.11)
//   n = 8, 1024 entries with aliasing outputs  2.049 -> 1.887 ms (FP64 tensor
//   pipe alone 0.70, HBM 0.98)
#include <algorithm>
#include <cstdint>

#include "kron_fibre.cuh"
#include "kron_launch.h"
#include "kron_mma8_core.cuh"
#include "kron_ptx.cuh"

namespace kron {

namespace {

using namespace ptx;

struct RingArgs
{
  void *base;           // base form: slot s at base + s stride
  long long stride;     // elements between slots
  void *const *ptrs;    // pointer form: slot s at ptrs[s]
  int slots, lag;
  unsigned magic;       // ceil(2^32 / slots): g / slots = umulhi(g, magic)
  int nentries;
  int *status;
  long long spin;
};

// Control words, each on a 128-byte line of its own: blocks that wait for one
// do not slow the atomics on the others.
constexpr int CTL_LINE = 32, CTL_QUEUE = 0, CTL_ABORT = CTL_LINE;
__host__ __device__ constexpr int ctl_phase1(int slot) { return (2 + 2 * slot) * CTL_LINE; }
__host__ __device__ constexpr int ctl_phase2(int slot) { return (3 + 2 * slot) * CTL_LINE; }
constexpr int RING_MAX_SLOTS = 512;
static_assert(ctl_phase1(RING_MAX_SLOTS) <= 6 * 6 * 6 * 6 * 6 * 6, "they fit a workspace vector");

template <typename T>
__device__ __forceinline__ T *ring_slot(const RingArgs &w, int s)
{
  return w.ptrs ? static_cast<T *>(w.ptrs[s]) : static_cast<T *>(w.base) + (long long)s * w.stride;
}

template <typename T>
__device__ __forceinline__ int *ring_ctl(const RingArgs &w)
{
  return reinterpret_cast<int *>(ring_slot<T>(w, w.slots));
}

template <typename T>
__global__ void ring_init_kernel(const __grid_constant__ RingArgs w)
{
  int *c = ring_ctl<T>(w);
  for (int i = threadIdx.x; i < ctl_phase1(w.slots); i += blockDim.x)
    c[i] = 0;
}

__device__ __forceinline__ int ld_relaxed(const int *p)
{
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_relaxed(int *p)
{
  asm volatile("red.relaxed.gpu.global.add.s32 [%0], 1;" ::"l"(p) : "memory");
}

// W is read by other blocks than wrote it and is written anew a ring later:
// loads and stores go to the L2 cache, where evict-last keeps the ring while
// x and y (evict-first) stream past
struct RingPol
{
  uint64_t keep, stream;
};

__device__ __forceinline__ RingPol ring_policies()
{
  RingPol p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p.keep));
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p.stream));
  return p;
}

__device__ __forceinline__ void w_store(double *p, double v, uint64_t pol)
{
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void w_store(float *p, float v, uint64_t pol)
{
  asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ double w_load(const double *p, uint64_t pol)
{
  double v;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.f64 %0, [%1], %2;"
               : "=d"(v)
               : "l"(p), "l"(pol)
               : "memory");
  return v;
}
__device__ __forceinline__ float w_load(const float *p, uint64_t pol)
{
  float v;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.f32 %0, [%1], %2;"
               : "=f"(v)
               : "l"(p), "l"(pol)
               : "memory");
  return v;
}
__device__ __forceinline__ void y_add(double *p, double v, uint64_t pol)
{
  asm volatile("red.global.add.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void y_add(float *p, float v, uint64_t pol)
{
  asm volatile("red.global.add.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol)
               : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, uint64_t pol)
{
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)),
                 "l"(src), "l"(pol)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %3, %2;" ::"r"(smem_addr(dst)),
                 "l"(src), "l"(pol), "n"(BYTES)
                 : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src),
               "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// What a block knows of an item, in shared memory.
struct Item
{
  int idx;              // queue position (>= the total: no more work)
  int ok;               // both dependencies were met when they were looked at
  int slot1, slot2;     // ring slots of phase 1 and phase 2, -1: no such part
  int need1, need2;     // counts that the slots' counters must have reached
  // 0-5: A_1..A_6 of the phase-1 entry, 6: its x, 7: its ring slot,
  // 8-13: A_1..A_6 of the phase-2 entry, 14: its y, 15: its ring slot
  void *ptr[16];
};

// The item of queue position idx, all but the pointers (one thread).
template <int K>
__device__ __forceinline__ void item_plan(Item &it, int idx, int total, const RingArgs &w)
{
  it.idx   = idx;
  it.ok    = 0;
  it.slot1 = it.slot2 = -1;
  if (idx >= total)
    return;
  const int g1 = idx / K, g2 = g1 - w.lag;
  if (g1 < w.nentries)
  {
    const int gen = (int)__umulhi((unsigned)g1, w.magic);
    it.slot1      = g1 - gen * w.slots;
    it.need1      = gen * K;
  }
  if (g2 >= 0)
  {
    const int gen = (int)__umulhi((unsigned)g2, w.magic);
    it.slot2      = g2 - gen * w.slots;
    it.need2      = (gen + 1) * K;
  }
}

// The queue side of a block: item i in slot i % 3 of `items`, fetched two
// items ahead by warp 0, a step at a time (the position when an item begins,
// the pointers in its middle, the slot at its end).  Lane j < 16 of the warp
// fetches pointer j, at base + index * stride, or what is stored there.
template <typename T, int K>
struct RingQueue
{
  Item *items;
  int *s_dead;
  int *ctl;
  int total;
  const char *base;  // warp 0
  long long stride;
  bool indirect;
  int qn;            // lane 0: the queue position taken last
  const void *pn;    // a pointer in flight
  int pub1, pub2;    // thread 0: slots whose parts of the last item are unpublished

  __device__ __forceinline__ const void *pointer(int lane, int idx, const RingArgs &w)
  {
    int g = idx / K - (lane < 8 ? 0 : w.lag);
    if (lane >= 16 || idx >= total || g < 0 || g >= w.nentries)
      return nullptr;
    if ((lane & 7) == 7)
      g -= (int)__umulhi((unsigned)g, w.magic) * w.slots;
    const char *a = base + g * stride;
    return indirect ? *reinterpret_cast<const void *const *>(a) : a;
  }
  __device__ __forceinline__ void start(const Params &p, const RingArgs &w, int tid)
  {
    ctl   = ring_ctl<T>(w);
    total = (w.nentries + w.lag) * K;
    pub1 = pub2 = -1;
    if (tid < 32)
    {
      int q0 = 0, q1 = 0;
      if (tid == 0)
      {
        q0 = atomicAdd(ctl + CTL_QUEUE, 2);
        q1 = q0 + 1;
        item_plan<K>(items[0], q0, total, w);
        item_plan<K>(items[1], q1, total, w);
      }
      const int m = tid & 7;
      if (m == 7)
      {
        indirect = w.ptrs != nullptr;
        base     = reinterpret_cast<const char *>(indirect ? (const void *)w.ptrs : w.base);
        stride   = indirect ? 8 : w.stride * (long long)sizeof(T);
      }
      else if (m == 6)
      {
        indirect = p.layout != LAYOUT_BATCHED;
        if (indirect)
          base = tid < 8 ? reinterpret_cast<const char *>(p.pX)
                         : reinterpret_cast<const char *>(p.pY);
        else
          base = static_cast<const char *>(tid < 8 ? p.X : p.Y);
        stride = indirect ? 8
                          : (tid < 8 ? p.xstride : p.ystride) * (long long)sizeof(T);
        base += p.ebase * stride;
      }
      else
      {
        indirect = p.layout != LAYOUT_BATCHED && p.layout != LAYOUT_PBATCHED;
        const long long nn = (long long)p.n[0] * p.n[0] * (long long)sizeof(T);
        stride   = indirect ? 8LL * p.apk : 6 * nn;
        base     = indirect ? reinterpret_cast<const char *>(p.pA) + 8 * m
                            : static_cast<const char *>(p.A) + m * nn;
        base += p.ebase * stride;
      }
      q0 = __shfl_sync(0xffffffffu, q0, 0);
      q1 = __shfl_sync(0xffffffffu, q1, 0);
      const void *p0 = pointer(tid, q0, w), *p1 = pointer(tid, q1, w);
      if (tid < 16)
      {
        items[0].ptr[tid] = const_cast<void *>(p0);
        items[1].ptr[tid] = const_cast<void *>(p1);
      }
    }
    if (tid == 0)
      *s_dead = 0;
  }
  // item i begins: take the position of item i + 2
  __device__ __forceinline__ void take(int tid)
  {
    if (tid == 0)
      qn = atomicAdd(ctl + CTL_QUEUE, 1);
  }
  // mid-item, warp 0: the pointers of item i + 2 take off
  __device__ __forceinline__ void mid(const RingArgs &w, int tid)
  {
    if (tid < 32)
    {
      qn = __shfl_sync(0xffffffffu, qn, 0);
      pn = pointer(tid, qn, w);
    }
  }
  // thread 0, in the middle of an item, when the last item's accesses have
  // drained: publish that item's parts and look at the next item's
  // dependencies, under one fence
  __device__ __forceinline__ void publish(Item *next)
  {
    bool ok = true;
    if (next && next->idx < total)
    {
      const int *a = ctl + ctl_phase2(max(next->slot1, 0));
      const int *b = ctl + ctl_phase1(max(next->slot2, 0));
      const int va = ld_relaxed(a), vb = ld_relaxed(b);
      ok = (next->slot1 < 0 || va >= next->need1) && (next->slot2 < 0 || vb >= next->need2);
    }
    __threadfence();
    if (pub1 >= 0)
      red_relaxed(ctl + ctl_phase1(pub1));
    if (pub2 >= 0)
      red_relaxed(ctl + ctl_phase2(pub2));
    pub1 = pub2 = -1;
    if (next)
      next->ok = ok ? 1 : 0;
  }
  // late in item i: item i + 2 takes its slot (warp 0)
  __device__ __forceinline__ void late(Item &it, const RingArgs &w, int tid)
  {
    if (tid < 16)
      it.ptr[tid] = const_cast<void *>(pn);
    if (tid == 0)
      item_plan<K>(it, qn, total, w);
  }
  // whole block, for an item whose dependencies were not met: false when the
  // wait ran out (or another block's did)
  __device__ __forceinline__ bool wait(const Item &it, const RingArgs &w, int tid)
  {
    if (tid == 0)
    {
      publish(nullptr);
      const int *a = it.slot1 >= 0 ? ctl + ctl_phase2(it.slot1) : nullptr;
      const int *b = it.slot2 >= 0 ? ctl + ctl_phase1(it.slot2) : nullptr;
      long long polls = 0;
      int dead        = 0;
      while (true)
      {
        const int va = a ? ld_relaxed(a) : 0, vb = b ? ld_relaxed(b) : 0;
        if ((!a || va >= it.need1) && (!b || vb >= it.need2))
          break;
        ++polls;
        if (polls >= w.spin || (polls % 64 == 0 && ld_relaxed(ctl + CTL_ABORT) != 0))
        {
          dead = 1;
          if (w.status)
            atomicExch(w.status, 1);
          atomicExch(ctl + CTL_ABORT, 1);
          break;
        }
        __nanosleep(200);
      }
      __threadfence();
      *s_dead = dead;
    }
    __syncthreads();
    return *s_dead == 0;
  }
};

// ---------------------------------------------------------------------------
// CUDA-core form: tail = modes 3..6, head = modes 1, 2, all products on
// fibres of two modes in registers (n^2 elements and one factor).
//   phase 1, R head rows of n^4: the rows arrive by cp.async during the item
//   before; modes 5, 6 in place on contiguous fibres; modes 3, 4 on strided
//   fibres, results from registers into W;
//   phase 2: a thread takes a column, n^2 elements of W at stride n^4.
// Stage layout: fibre (chunk) c of n^2 contiguous elements at chunk_off(c),
// padded so that the 16-byte accesses of neighbouring lanes' chunks hit
// distinct banks (n = 6 FP64: 16 bytes after every fourth chunk; n = 8 FP32:
// after every chunk; the others' chunk lengths are odd in 16-byte or element
// units).
template <typename T, int N, int R_, int THREADS_>
struct RingShape
{
  static constexpr int N2 = N * N, LT = N2 * N2, LH = N2, L = LT * LH;
  static constexpr int R = R_, THREADS = THREADS_;
  static constexpr int K   = (LH + R - 1) / R;
  static constexpr int CPI = (LT + K - 1) / K;
  static constexpr int FIB = R * N2;
  static_assert(FIB <= THREADS && CPI <= THREADS, "one fibre a thread");
  static constexpr bool VEC   = N % 2 == 0; // chunks are whole 16-byte units
  static constexpr int V      = 16 / (int)sizeof(T);
  static constexpr int GROUP  = (N == 6 && sizeof(T) == 8) ? 4 : (N == 8 ? 1 : 0);
  static constexpr int ROW    = GROUP ? N2 * N2 + N2 / (GROUP ? GROUP : 1) * V : N2 * N2;
  static constexpr int BUF    = (R * ROW + 2 * V + 15) / 16 * 16; // + V: an unaligned start
  static constexpr int ASZ    = (6 * N2 + 3) / 4 * 4;             // A_1..A_6
  static constexpr size_t OFF_A    = 0;
  static constexpr size_t OFF_X    = 2 * (size_t)ASZ * sizeof(T);
  static constexpr size_t SMEM     = OFF_X + 2 * (size_t)BUF * sizeof(T);
  __device__ static constexpr int chunk_off(int c)
  {
    return c * N2 + (GROUP ? c / (GROUP ? GROUP : 1) * V : 0);
  }
};

template <typename T, int N, int R, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
    kron_ring_kernel(const __grid_constant__ Params p, const __grid_constant__ RingArgs w)
{
  using S          = RingShape<T, N, R, THREADS>;
  constexpr int N2 = S::N2, LT = S::LT, LH = S::LH, K = S::K, V = S::V;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Item s_item[3];
  __shared__ int s_dead;
  const int tid = threadIdx.x;
  auto stage_a  = [&](int b) { return reinterpret_cast<T *>(smem + S::OFF_A) + b * S::ASZ; };
  auto stage_x  = [&](int b) { return reinterpret_cast<T *>(smem + S::OFF_X) + b * S::BUF; };
  const RingPol pol = ring_policies();
  const int ld      = p.layout == LAYOUT_XBATCHED ? p.lda : N;

  // x rows and factors of item `it` into stage b.  A linear stage takes the
  // rows at the offset that their start has in a 16-byte unit.
  auto issue = [&](const Item &it, int b) {
    if (it.slot1 >= 0)
    {
      const int h0 = it.idx % K * R, ne = min(R, LH - h0) * LT;
      const T *src = static_cast<const T *>(it.ptr[6]) + (long long)h0 * LT;
      T *buf       = stage_x(b);
      if constexpr (S::VEC)
      {
        if (aligned16(src))
          for (int u = tid; u < ne / V; u += THREADS)
            cp_async<16>(buf + u * V + (S::chunk_off(u * V / N2) - u * V / N2 * N2), src + u * V,
                         pol.stream);
        else
          for (int u = tid; u < ne; u += THREADS)
            cp_async<sizeof(T)>(buf + u + (S::chunk_off(u / N2) - u / N2 * N2), src + u);
      }
      else
      {
        const int sh = (int)((reinterpret_cast<uintptr_t>(src) & 15) / sizeof(T));
        // units [u0, u1) lie whole in the rows; the ends go by elements
        const int u0 = (sh + V - 1) / V, u1 = (sh + ne) / V;
        for (int u = u0 + tid; u < u1; u += THREADS)
          cp_async<16>(buf + u * V, src - sh + u * V, pol.stream);
        if (tid < u0 * V - sh)
          cp_async<sizeof(T)>(buf + sh + tid, src + tid);
        else if (tid >= 32 && u1 * V + tid - 32 < sh + ne)
          cp_async<sizeof(T)>(buf + u1 * V + tid - 32, src + (u1 * V + tid - 32 - sh));
      }
    }
    T *as = stage_a(b);
    for (int q = tid; q < 6 * N2; q += THREADS)
    {
      // A_1, A_2 of the phase-2 entry, A_3..A_6 of the phase-1 entry
      const int l = q / N2, ij = q - l * N2, j = ij / N, i = ij - j * N;
      if (l < 2 ? it.slot2 >= 0 : it.slot1 >= 0)
        cp_async<sizeof(T)>(as + q, static_cast<const T *>(it.ptr[l < 2 ? 8 + l : l]) + i +
                                        (long long)j * ld);
    }
  };

  RingQueue<T, K> q;
  q.items  = s_item;
  q.s_dead = &s_dead;
  q.start(p, w, tid);
  __syncthreads();
  if (s_item[0].idx < q.total)
    issue(s_item[0], 0);
  cp_async_wait();
  __syncthreads();

  for (int i = 0;; ++i)
  {
    const int b     = i & 1;
    const Item &it  = s_item[i % 3];
    if (it.idx >= q.total)
      break;
    if (!it.ok && !q.wait(it, w, tid))
      break;
    Item &next     = s_item[(i + 1) % 3];
    const int part = it.idx % K;
    q.take(tid);
    if (next.idx < q.total)
      issue(next, b ^ 1);
    const T *as = stage_a(b);

    // ---- phase 1, modes 5 and 6 in place
    const bool p1  = it.slot1 >= 0;
    const int h0   = part * R;
    const int nfib = min(R, LH - h0) * N2;
    T *xs          = stage_x(b);
    if constexpr (!S::VEC)
      if (p1)
        xs += (reinterpret_cast<uintptr_t>(static_cast<const T *>(it.ptr[6]) +
                                           (long long)h0 * LT) & 15) / sizeof(T);
    if (p1 && tid < nfib)
    {
      T *c = xs + S::chunk_off(tid);
      T v[N2];
      load_chunk<T, N>(c, v);
      apply_fast<T, N>(v, as + 5 * N2);
      apply_slow<T, N>(v, as + 4 * N2);
      store_chunk<T, N>(c, v);
    }
    __syncthreads();
    q.mid(w, tid);
    if (tid == 0)
      q.publish(&next);
    // ---- phase 1, modes 3 and 4; results into W
    if (p1 && tid < nfib)
    {
      const int row = tid / N2, r = tid - row * N2;
      const T *c    = xs + row * S::ROW + r;
      T v[N2];
#pragma unroll
      for (int e = 0; e < N2; e++)
        v[e] = c[S::chunk_off(e)];
      apply_fast<T, N>(v, as + 3 * N2);
      apply_slow<T, N>(v, as + 2 * N2);
      T *wp = static_cast<T *>(it.ptr[7]) + (long long)(h0 + row) * LT + r;
#pragma unroll
      for (int e = 0; e < N2; e++)
        w_store(wp + e * N2, v[e], pol.keep);
    }
    // ---- phase 2, modes 1 and 2 on columns of W, added into y
    const int col = part * S::CPI + tid;
    if (it.slot2 >= 0 && tid < S::CPI && col < LT)
    {
      const T *wp = static_cast<const T *>(it.ptr[15]) + col;
      T v[N2];
#pragma unroll
      for (int e = 0; e < N2; e++)
        v[e] = w_load(wp + (long long)e * LT, pol.keep);
      apply_fast<T, N>(v, as + 1 * N2);
      apply_slow<T, N>(v, as + 0 * N2);
      T *y = static_cast<T *>(it.ptr[14]) + col;
#pragma unroll
      for (int e = 0; e < N2; e++)
        y_add(y + (long long)e * LT, v[e], pol.stream);
    }
    q.pub1 = it.slot1;
    q.pub2 = it.slot2;
    q.late(s_item[(i + 2) % 3], w, tid);
    cp_async_wait();
    __syncthreads();
  }
  if (tid == 0)
    q.publish(nullptr);
}

// ---------------------------------------------------------------------------
// Tensor-core form (FP64, n = 7 and 8; n = 7 zero padded to 8): head = modes
// 1..3, tail = modes 4..6, everything in mma.sync f64 fragments.
//   phase 1: a warp takes a head row of n^3 elements (brought into its row
//   buffer by cp.async during the item before), applies the three tail modes
//   (kron8x3_tile) and stores the result into W;
//   phase 2: a block takes 8 columns of W.  Warp j_1 loads its (j_2, j_3) x 8
//   columns (64-byte row segments) with the columns on the fragments' G index
//   and applies modes 3 and 2; the results change hands through shared memory
//   (E[j_1][i_2][i_3][c]); warp i_2 applies mode 1 and adds into y.
// E's strides spread the eight columns of four quads over distinct banks for
// both its writes (i_2 = 2t+p) and its reads (j_1 = 2t+p).  A warp's slice of
// E is also its transpose scratch.
template <int N>
struct RingMma
{
  static constexpr int N3 = N * N * N, L = N3 * N3;
  static constexpr int K  = (N3 + 7) / 8;
  static constexpr int THREADS = 256, MINB = 2;
  static constexpr int S2 = 66, S1 = 8 * S2 + 2; // strides of E's i_2 and j_1
  static constexpr int ASZ = 6 * N * N;
  static constexpr size_t OFF_E = (2 * (size_t)ASZ * 8 + 15) / 16 * 16;
  // a warp's head row, at the offset that its start has in a 16-byte unit
  static constexpr int ROW      = (N3 + 2 + 1) / 2 * 2;
  static constexpr size_t OFF_X = OFF_E + 8 * (size_t)S1 * 8;
  static constexpr size_t SMEM  = OFF_X + 8 * (size_t)ROW * 8;
};

template <int N>
__device__ __forceinline__ void frag_of(double (&b)[2], const double *A, int g, int t)
{
#pragma unroll
  for (int s = 0; s < 2; s++)
    b[s] = (N == 8 || (g < N && 2 * t + s < N)) ? A[g + (2 * t + s) * N] : 0.0;
}

template <int N>
__global__ void __launch_bounds__(RingMma<N>::THREADS, RingMma<N>::MINB)
    kron_ring_mma_kernel(const __grid_constant__ Params p, const __grid_constant__ RingArgs w)
{
  using S          = RingMma<N>;
  constexpr int N2 = N * N, N3 = S::N3, K = S::K;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Item s_item[3];
  __shared__ int s_dead;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  double *E       = reinterpret_cast<double *>(smem + S::OFF_E);
  double *scratch = E + warp * S::S1;
  auto stage_a    = [&](int b) { return reinterpret_cast<double *>(smem) + b * S::ASZ; };
  const RingPol pol = ring_policies();
  const int ld      = p.layout == LAYOUT_XBATCHED ? p.lda : N;

  auto issue_a = [&](const Item &it, int b) {
    double *as = stage_a(b);
    for (int q = tid; q < 6 * N2; q += S::THREADS)
    {
      // A_1..A_3 of the phase-2 entry, A_4..A_6 of the phase-1 entry
      const int l = q / N2, ij = q - l * N2, j = ij / N, i = ij - j * N;
      if (l < 3 ? it.slot2 >= 0 : it.slot1 >= 0)
        cp_async<8>(as + q, static_cast<const double *>(it.ptr[l < 3 ? 8 + l : l]) + i +
                                (long long)j * ld);
    }
  };
  // this warp's head row of `it` into its row buffer
  double *row    = reinterpret_cast<double *>(smem + S::OFF_X) + warp * S::ROW;
  auto issue_row = [&](const Item &it) {
    const int h = it.idx % K * 8 + warp;
    if (it.slot1 < 0 || h >= N3)
      return;
    const double *x = static_cast<const double *>(it.ptr[6]) + (long long)h * N3;
    const int sh    = aligned16(x) ? 0 : 1;
    const int u1    = (sh + N3) / 2; // units [sh, u1) lie whole in the row
    for (int u = sh + lane; u < u1; u += 32)
      cp_async<16>(row + 2 * u, x - sh + 2 * u, pol.stream);
    if (sh && lane == 0)
      cp_async<8>(row + 1, x);
    if (((sh + N3) & 1) && lane == 1)
      cp_async<8>(row + 2 * u1, x + N3 - 1);
  };

  RingQueue<double, K> q;
  q.items  = s_item;
  q.s_dead = &s_dead;
  q.start(p, w, tid);
  __syncthreads();
  if (s_item[0].idx < q.total)
  {
    issue_a(s_item[0], 0);
    issue_row(s_item[0]);
  }
  cp_async_wait();
  __syncthreads();

  for (int i = 0;; ++i)
  {
    const int b    = i & 1;
    const Item &it = s_item[i % 3];
    if (it.idx >= q.total)
      break;
    if (!it.ok && !q.wait(it, w, tid))
      break;
    Item &next     = s_item[(i + 1) % 3];
    const int part = it.idx % K;
    q.take(tid);
    const double *as = stage_a(b);
    // ---- phase 2: this warp's (j_2, j_3) of eight columns, j_1 = warp,
    // columns c = g (on their way during phase 1)
    const int col  = part * 8 + g;
    const bool own = it.slot2 >= 0 && warp < N;
    double wv[8][2];
    if (own)
    {
      const double *wp = static_cast<const double *>(it.ptr[15]) + (long long)warp * N2 * N3 + col;
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
        {
          wv[qq][s] = 0.0;
          if (N == 8 || (qq < N && 2 * t + s < N && col < N3))
            wv[qq][s] = w_load(wp + (long long)(qq * N + 2 * t + s) * N3, pol.keep);
        }
    }
    // ---- phase 1: modes 6, 5, 4 on head row h -> W
    const int h = part * 8 + warp;
    if (it.slot1 >= 0 && h < N3)
    {
      AFrag8 f;
      frag_of<N>(f.b1, as + 3 * N2, g, t);
      frag_of<N>(f.b2, as + 4 * N2, g, t);
      frag_of<N>(f.a3, as + 5 * N2, g, t);
      double v[8][2], acc[8][2];
      const bool odd = !aligned16(static_cast<const double *>(it.ptr[6]) + (long long)h * N3);
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
      {
        const double *src = row + (odd ? 1 : 0) + qq * N2 + g * N + 2 * t;
        if (N == 8 && !odd)
        {
          const double2 u = *reinterpret_cast<const double2 *>(src);
          v[qq][0]        = u.x;
          v[qq][1]        = u.y;
        }
        else
#pragma unroll
          for (int s = 0; s < 2; s++)
            v[qq][s] = (N == 8 || (qq < N && g < N && 2 * t + s < N)) ? src[s] : 0.0;
        acc[qq][0] = acc[qq][1] = 0.0;
      }
      kron8x3_tile<N>(v, acc, f, scratch, g, t);
      if (tid == 0)
        q.publish(&next);
      double *wp = static_cast<double *>(it.ptr[7]) + (long long)h * N3;
#pragma unroll
      for (int qq = 0; qq < N; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
          if (N == 8 || (g < N && 2 * t + s < N))
            w_store(wp + (2 * t + s) * N2 + qq * N + g, acc[qq][s], pol.keep);
    }
    else if (tid == 0)
      q.publish(&next);
    // the next item's row and factors
    __syncwarp(); // the row buffer is read
    q.mid(w, tid);
    if (next.idx < q.total)
    {
      issue_a(next, b ^ 1);
      issue_row(next);
    }
    // ---- phase 2, modes 3 and 2
    if (own)
    {
      double b3[2], b2[2], r[8][2];
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
        r[qq][0] = r[qq][1] = 0.0;
      frag_of<N>(b3, as + 2 * N2, g, t);
      frag_of<N>(b2, as + 1 * N2, g, t);
      mma_along_p(wv, r, b3);
      if (N < 8)
        r[7][0] = r[7][1] = 0.0; // j_2 = 7
      quad_transpose(r, wv, scratch, g, t);
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
        r[qq][0] = r[qq][1] = 0.0;
      mma_along_p(wv, r, b2);
      __syncwarp(); // the scratch is read; the slice takes the results
#pragma unroll
      for (int qq = 0; qq < N; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
          scratch[(2 * t + s) * S::S2 + qq * 8 + g] = r[qq][s];
    }
    __syncthreads();
    // ---- phase 2, mode 1: warp = i_2
    if (own)
    {
      double b1[2], v[8][2], r[8][2];
      frag_of<N>(b1, as, g, t);
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
        {
          v[qq][s] = (qq < N && (N == 8 || 2 * t + s < N))
                         ? E[(2 * t + s) * S::S1 + warp * S::S2 + qq * 8 + g]
                         : 0.0;
          r[qq][s] = 0.0;
        }
      mma_along_p(v, r, b1);
      double *y = static_cast<double *>(it.ptr[14]) + (long long)warp * N * N3 + col;
#pragma unroll
      for (int qq = 0; qq < N; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
          if (N == 8 || (2 * t + s < N && col < N3))
            y_add(y + (long long)((2 * t + s) * N2 + qq) * N3, r[qq][s], pol.stream);
    }
    q.pub1 = it.slot1;
    q.pub2 = it.slot2;
    q.late(s_item[(i + 2) % 3], w, tid);
    cp_async_wait();
    __syncthreads();
  }
  if (tid == 0)
    q.publish(nullptr);
}

// ---------------------------------------------------------------------------
// Vectors of W the call may use, the control words' among them.
template <typename T>
int ring_workspace(const Params &p, const Workspace &wsp, long long L, RingArgs &w)
{
  long long have = 0;
  if (p.layout == LAYOUT_BATCHED)
  {
    if (!wsp.W || wsp.wstride < L)
      return KRON_ERROR_WORKSPACE;
    have     = p.eend - p.ebase;
    w.base   = static_cast<T *>(wsp.W);
    w.stride = wsp.wstride;
  }
  else if (wsp.pW)
  {
    if (wsp.pw_elems < L)
      return KRON_ERROR_WORKSPACE;
    have   = wsp.npW;
    w.ptrs = wsp.pW;
  }
  else
  {
    have     = wsp.W ? (long long)(wsp.Wbytes / (sizeof(T) * (size_t)L)) : 0;
    w.base   = wsp.W;
    w.stride = L;
  }
  if (have < 3)
    return KRON_ERROR_WORKSPACE;
  w.slots = (int)std::min<long long>(have - 1, RING_MAX_SLOTS);
  return KRON_SUCCESS;
}

template <typename T>
int ring_launch(const void *fn, int threads, size_t smem, int K, long long L, int ahead, Params p,
                const Workspace &wsp, cudaStream_t stream)
{
  RingArgs w{};
  const int rc = ring_workspace<T>(p, wsp, L, w);
  if (rc != KRON_SUCCESS)
    return rc;
  int per_sm = 1;
  if (cached_occupancy(fn, threads, smem, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  w.nentries = p.eend - p.ebase;
  w.status   = device_status_ptr();
  w.spin     = wait_limit();
  const long long blocks = (long long)device_info().sms * per_sm;
  // `ahead` items of every block between an entry's phases, and as many until
  // its slot is written again
  const int groups = (int)(ahead * blocks / K + 1);
  w.lag            = std::max(1, std::min({groups, w.nentries, w.slots - 1}));
  w.slots          = std::min(w.slots, w.lag + groups);
  w.magic            = (unsigned)(((1ULL << 32) + w.slots - 1) / w.slots);
  const long long items = (long long)(w.nentries + w.lag) * K;
  // 32-bit queue positions (two a block taken beyond the end), and the range
  // in which the division by `slots` is exact
  if (items + 3 * blocks > 2147000000LL ||
      ((long long)w.nentries + w.lag) * w.slots >= (1LL << 32))
    return KRON_ERROR_NOT_SUPPORTED;
  ring_init_kernel<T><<<1, 128, 0, stream>>>(w);
  void *args[] = {&p, &w};
  return cudaLaunchKernel(fn, dim3((unsigned)std::min(blocks, items)), dim3(threads), args, smem,
                          stream) == cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

template <typename T, int N, int R, int THREADS, int MINB>
int launch_ring_t(const Params &p, const Workspace &wsp, cudaStream_t stream)
{
  using S = RingShape<T, N, R, THREADS>;
  return ring_launch<T>(reinterpret_cast<const void *>(&kron_ring_kernel<T, N, R, THREADS, MINB>),
                        THREADS, S::SMEM, S::K, S::L, 2, p, wsp, stream);
}

template <int N>
int launch_ring_mma(const Params &p, const Workspace &wsp, cudaStream_t stream)
{
  using S = RingMma<N>;
  return ring_launch<double>(reinterpret_cast<const void *>(&kron_ring_mma_kernel<N>), S::THREADS,
                             S::SMEM, S::K, S::L, 3, p, wsp, stream);
}

} // namespace

bool ring_supported(const Params &p, int prec)
{
  if ((prec != PREC_F64 && prec != PREC_F32) || p.seg_off ||
      (p.accum != ACC_DISTINCT && p.accum != ACC_ATOMIC) || p.d != 6)
    return false;
  const int n = p.n[0];
  for (int l = 0; l < p.d; l++)
    if (p.m[l] != n || p.n[l] != n)
      return false;
  return n >= 6 && n <= 8;
}

int launch_ring(const Params &p, int prec, const Workspace &ws, cudaStream_t stream)
{
  if (p.eend <= p.ebase)
    return KRON_SUCCESS;
  const int n = p.n[0];
  if (prec == PREC_F32)
    return n == 7   ? launch_ring_t<float, 7, 5, 256, 2>(p, ws, stream)
           : n == 8 ? launch_ring_t<float, 8, 2, 128, 3>(p, ws, stream)
                    : KRON_ERROR_NOT_SUPPORTED;
  return n == 6   ? launch_ring_t<double, 6, 3, 128, 3>(p, ws, stream)
         : n == 7 ? launch_ring_mma<7>(p, ws, stream)
                  : launch_ring_mma<8>(p, ws, stream);
}

} // namespace kron
