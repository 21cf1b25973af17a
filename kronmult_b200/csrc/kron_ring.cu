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
// its entry's K phase-1 parts, lag entries back (normally long done), and
// phase 1 for the ring slot of W it writes, last read by the entry `slots`
// positions back.  W is a ring of `slots` vectors, a few tens of MB however
// large the batch, most of it in the L2 cache (0.8 of its 3.1 GB of stores and
// loads go to DRAM for 4096 entries of n = 6, 2.4 of 4.3 GB for 1024 of n = 8);
// no cluster barriers, and every SM works on both phases, so loads of x, math
// and adds into y overlap between the blocks of an SM.
//
// The control words (queue, abort, and per slot the parts done of each phase,
// counted up over the slot's generations) lie in the workspace vector after
// the ring, zeroed by a small kernel ahead of this one.  Waits are bounded
// (wait_limit() polls): a group that gives up records 1 in the device status
// word, raises the abort word, which ends the others' waits, and leaves as a
// whole once its copies have landed; y of the parts not done is untouched.
//
// Measured against what ran before (the cluster two-phase kernel, whose W
// goes through HBM and back: 9.35 against 6.87 GB for 1024 entries of n = 8;
// n = 6: the slab-cluster kernel with its side kernel):
//   n = 6, 4096 entries  1.40 -> 1.20 ms (HBM alone 0.70)
//   n = 7, 256 entries   0.466 -> 0.250 ms (HBM alone 0.11)
//   n = 8, 1024 entries with aliasing outputs  2.05 -> 1.79 ms (FP64 tensor
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

// What a block knows of an item, in shared memory.
struct Item
{
  int idx;              // queue position (>= the total: no more work)
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

// ---------------------------------------------------------------------------
// Control warps, beside the group of warps that compute (a block, or a third of
// one).  One takes items from the queue, starts their copies and waits for their
// dependencies, an item ahead of the computing warps; another publishes parts,
// so that its fences (2-3 us behind adds into y) hold nobody up.  Slot s
// of two holds an item's operands; mbarriers:
//   full[s]  the copies have landed (an arrival of each lane) and the
//            dependencies are met (lane 0's).
// Descriptions have four slots, so that the taker need not wait for the
// publisher:
//   done[d]  an arrival of each computing warp, behind its last access (of the
//            taker in their place, for the end of the queue);
//   read[d]  the publisher has read description d.
// (No barrier can run two phases ahead of a thread that waits for it.)
// All waits are bounded.  When one of the taker's runs out, it raises the status
// and abort words and the computing warps find the end of the queue.  When one
// of the computing warps' does, that warp raises them and `left`, and the group's
// warps leave together at the item's barrier, which carries their vote (a warp
// that left alone would leave the others at the barrier for ever); `left` ends
// the waits of the taker and the publisher for them.  Who leaves early first lets
// the copies that it waits for or started land.
constexpr int ITEM_SLOTS = 4;
struct ControlBars
{
  uint64_t full[2], done[ITEM_SLOTS], read[ITEM_SLOTS];
  int left; // the computing warps have given up
};

// one thread, before the block's first barrier; `warps` that compute
__device__ __forceinline__ void control_init(ControlBars &bars, int warps)
{
  for (int s = 0; s < 2; s++)
    mbar_init(&bars.full[s], 33);
  for (int d = 0; d < ITEM_SLOTS; d++)
  {
    mbar_init(&bars.done[d], warps);
    mbar_init(&bars.read[d], 1);
  }
  bars.left = 0;
}

// the group's computing warps have left, or are about to
__device__ __forceinline__ bool has_left(const ControlBars &bars)
{
  return *reinterpret_cast<const volatile int *>(&bars.left) != 0;
}

// A barrier of THREADS threads (whole warps) that ANDs what they bring.
template <int THREADS>
__device__ __forceinline__ bool vote_sync(int id, bool v)
{
  int all;
  asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n"
               " bar.red.and.pred q, %2, %3, p;\n selp.s32 %0, 1, 0, q;\n}"
               : "=r"(all)
               : "r"((int)v), "r"(id), "n"(THREADS)
               : "memory");
  return all != 0;
}

// a bulk copy of this lane's that full[s] waits for
__device__ __forceinline__ void bulk_into(uint64_t *bar, void *dst, const void *src, int bytes,
                                          uint64_t pol)
{
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
               "[%0], [%1], %2, [%3], %4;" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(pol)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

template <typename T, int K>
struct RingControl
{
  // one thread
  static __device__ __forceinline__ void raise(const RingArgs &w)
  {
    if (w.status)
      atomicExch(w.status, 1);
    atomicExch(ring_ctl<T>(w) + CTL_ABORT, 1);
  }

  // one thread: the copies of item j, whose mbarrier has its arrivals, land
  static __device__ __forceinline__ void land(ControlBars &bars, int j, long long drain)
  {
    mbar_wait_bounded(&bars.full[j & 1], (j >> 1) & 1, drain);
  }

  // a computing warp whose wait for item i has run out, ahead of the vote
  static __device__ __forceinline__ void leave(const RingArgs &w, ControlBars &bars, int i,
                                            long long drain)
  {
    raise(w);
    *reinterpret_cast<volatile int *>(&bars.left) = 1;
    land(bars, i, drain);
  }

  // a wait for the computing warps, over when those have left
  static __device__ __forceinline__ bool wait_alive(uint64_t *bar, unsigned parity,
                                                    const ControlBars &bars, long long limit)
  {
    for (long long polls = 0; polls < limit; polls++)
    {
      if (mbar_try_wait(bar, parity))
        return true;
      if (has_left(bars))
        return false;
    }
    return false;
  }

  // one warp, beside `warps` that compute; issue(item, slot, full) starts the
  // copies of an item (whole warp)
  template <typename Issue>
  static __device__ __forceinline__ void run(const Params &p, const RingArgs &w, Item *items,
                                             ControlBars &bars, int warps, int lane,
                                             long long drain, const Issue &issue)
  {
    constexpr unsigned FULL = 0xffffffffu;
    int *ctl        = ring_ctl<T>(w);
    const int total = (w.nentries + w.lag) * K;
    // lane j < 16 finds pointer j at base + index * stride, or stored there
    const char *base = nullptr;
    long long stride = 0;
    bool indirect    = false;
    const int m      = lane & 7;
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
        base = lane < 8 ? reinterpret_cast<const char *>(p.pX)
                        : reinterpret_cast<const char *>(p.pY);
      else
        base = static_cast<const char *>(lane < 8 ? p.X : p.Y);
      stride = indirect ? 8 : (lane < 8 ? p.xstride : p.ystride) * (long long)sizeof(T);
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
    int q = 0;
    if (lane == 0)
      q = atomicAdd(ctl + CTL_QUEUE, 1);
    for (int j = 0;; j++)
    {
      constexpr int D = ITEM_SLOTS;
      Item &it      = items[j % D];
      uint64_t *bar = &bars.full[j & 1];
      const int idx = __shfl_sync(FULL, q, 0);
      bool ok       = (j < 2 || wait_alive(&bars.done[(j - 2) % D], ((j - 2) / D) & 1, bars, drain)) &&
                (j < D || mbar_wait_bounded(&bars.read[j % D], (j / D - 1) & 1, drain));
      ok = __all_sync(FULL, ok);
      if (!ok)
      {
        // nothing of this item was started, and the mbarrier it would use may
        // still be that of item j - 2; computing warps that have not left run
        // into their bound
        if (lane == 0)
        {
          raise(w);
          if (j > 1)
            land(bars, j - 2, drain);
          if (j > 0)
            land(bars, j - 1, drain);
        }
        return;
      }
      if (lane == 0 && idx < total)
        q = atomicAdd(ctl + CTL_QUEUE, 1);
      if (lane == 0)
        item_plan<K>(it, idx, total, w);
      if (lane < 16)
      {
        int g         = idx / K - (lane < 8 ? 0 : w.lag);
        const void *a = nullptr;
        if (idx < total && g >= 0 && g < w.nentries)
        {
          if (m == 7)
            g -= (int)__umulhi((unsigned)g, w.magic) * w.slots;
          a = base + g * stride;
          if (indirect)
            a = *static_cast<const void *const *>(a);
        }
        it.ptr[lane] = const_cast<void *>(a);
      }
      // the slot's last readers come before the copies
      fence_proxy_async();
      __syncwarp();
      const bool end = idx >= total;
      if (!end)
        issue(it, j & 1, bar);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar))
                   : "memory");
      bool met = true;
      if (!end)
      {
        const int *a = it.slot1 >= 0 ? ctl + ctl_phase2(it.slot1) : nullptr;
        const int *b = it.slot2 >= 0 ? ctl + ctl_phase1(it.slot2) : nullptr;
        for (long long polls = 0;; polls++)
        {
          // every lane reads: one transaction, and no divergence
          const int va = a ? ld_relaxed(a) : 0, vb = b ? ld_relaxed(b) : 0;
          met          = __all_sync(FULL, (!a || va >= it.need1) && (!b || vb >= it.need2));
          if (met || polls + 1 >= w.spin ||
              (polls % 64 == 63 && __any_sync(FULL, ld_relaxed(ctl + CTL_ABORT) != 0)))
            break;
          __nanosleep(100);
        }
        __threadfence(); // what the others published is visible from here on
      }
      if (!met && lane == 0)
      {
        raise(w);
        it.idx = total;
      }
      if (lane == 0)
        mbar_arrive(bar);
      if (end || !met)
      {
        if (lane == 0) // for the publisher
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&bars.done[j % D])),
                       "r"(warps)
                       : "memory");
        if (!met && lane == 0) // computing warps that have left wait for no copy of this item
          land(bars, j, drain);
        return;
      }
    }
  }

  // One thread: publishes the parts of item j of a group once its computing
  // warps are done with it.  0: not yet, 1: published, -1: the end of the queue,
  // or they have left without it.
  static __device__ __forceinline__ int publish(const RingArgs &w, const Item *items,
                                                ControlBars &bars, int j, int total)
  {
    if (!mbar_try_wait(&bars.done[j % ITEM_SLOTS], (j / ITEM_SLOTS) & 1))
      return has_left(bars) ? -1 : 0;
    const Item &it = items[j % ITEM_SLOTS];
    if (it.idx >= total)
      return -1;
    int *ctl     = ring_ctl<T>(w);
    const int s1 = it.slot1, s2 = it.slot2;
    mbar_arrive(&bars.read[j % ITEM_SLOTS]);
    __threadfence();
    if (s1 >= 0)
      red_relaxed(ctl + ctl_phase1(s1));
    if (s2 >= 0)
      red_relaxed(ctl + ctl_phase2(s2));
    return 1;
  }
  // the same for `groups` groups until all of them have come to the end
  static __device__ __forceinline__ void publish_all(const RingArgs &w, const Item (*items)[ITEM_SLOTS],
                                                     ControlBars *bars, int groups,
                                                     long long drain)
  {
    const int total = (w.nentries + w.lag) * K;
    int j[4] = {0, 0, 0, 0};
    unsigned open = (1u << groups) - 1;
    for (long long idle = 0; open && idle < drain; idle++)
#pragma unroll
      for (int g = 0; g < 4; g++)
        if (g < groups && (open >> g & 1))
        {
          const int r = publish(w, items[g], bars[g], j[g], total);
          if (r > 0)
          {
            j[g]++;
            idle = 0;
          }
          else if (r < 0)
            open &= ~(1u << g);
        }
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
//
// A block is three such groups of four warps, which share nothing but the
// control warps: three takers and a publisher.  One block an SM; the computing
// warps take the registers that the control warps leave (160 of 128 + 128 / 3 a
// thread: a fibre and a factor of n = 6 in FP64 are 144).  Spill
// stores are 48 bytes a thread there, 100 and 12 for n = 7, 8 in FP32.
template <typename T, int N, int R_>
struct RingShape
{
  static constexpr int N2 = N * N, LT = N2 * N2, LH = N2, L = LT * LH;
  static constexpr int R = R_, G = 128, GROUPS = 3, THREADS = 512;
  static constexpr int K   = (LH + R - 1) / R;
  static constexpr int CPI = (LT + K - 1) / K;
  static_assert(R * N2 <= G && CPI <= G, "one fibre a thread");
  // setmaxnreg: the shares of a launch with 128 registers a thread
  static constexpr int REGS = 160, CONTROL_REGS = 32;
  static_assert(3 * G * REGS + G * CONTROL_REGS <= THREADS * 128, "register shares");
  static constexpr bool VEC   = N % 2 == 0; // chunks are whole 16-byte units
  static constexpr int V      = 16 / (int)sizeof(T);
  static constexpr int GROUP  = (N == 6 && sizeof(T) == 8) ? 4 : (N == 8 ? 1 : 0);
  static constexpr int ROW    = GROUP ? N2 * N2 + N2 / (GROUP ? GROUP : 1) * V : N2 * N2;
  static constexpr int BUF    = (R * ROW + 2 * V + 15) / 16 * 16; // + V: an unaligned start
  static constexpr int ASZ    = (6 * N2 + 3) / 4 * 4;             // A_1..A_6
  static constexpr int STAGE  = ASZ + BUF;                        // elements, two a group
  static constexpr size_t SMEM = GROUPS * 2 * (size_t)STAGE * sizeof(T);
  __device__ static constexpr int chunk_off(int c)
  {
    return c * N2 + (GROUP ? c / (GROUP ? GROUP : 1) * V : 0);
  }
};

template <typename T, int N, int R>
__global__ void __launch_bounds__(RingShape<T, N, R>::THREADS, 1)
    kron_ring_kernel(const __grid_constant__ Params p, const __grid_constant__ RingArgs w,
                     long long drain)
{
  using S          = RingShape<T, N, R>;
  constexpr int N2 = S::N2, LT = S::LT, LH = S::LH, K = S::K, V = S::V;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Item s_item[S::GROUPS][ITEM_SLOTS];
  __shared__ ControlBars s_bars[S::GROUPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // stage b of group gr: A_1..A_6, then the rows
  auto stage_a = [&](int gr, int b) {
    return reinterpret_cast<T *>(smem) + (gr * 2 + b) * S::STAGE;
  };
  const RingPol pol = ring_policies();
  const int total   = (w.nentries + w.lag) * K;
  if (threadIdx.x == 0)
  {
    for (int gr = 0; gr < S::GROUPS; gr++)
      control_init(s_bars[gr], 4);
    fence_mbar_init();
  }
  __syncthreads();

  if (warp >= 4 * S::GROUPS)
  {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::CONTROL_REGS));
    const int gr = warp - 4 * S::GROUPS;
    if (gr == S::GROUPS)
    {
      if (lane == 0)
        RingControl<T, K>::publish_all(w, s_item, s_bars, S::GROUPS, drain);
      return;
    }
    const int ld = p.layout == LAYOUT_XBATCHED ? p.lda : N;
    // x rows and factors of an item; a linear stage takes the rows at the
    // offset that their start has in a 16-byte unit
    RingControl<T, K>::run(p, w, s_item[gr], s_bars[gr], 4, lane, drain, [&](const Item &it, int b,
                                                                          uint64_t *bar) {
      T *as = stage_a(gr, b);
      // A_1, A_2 of the phase-2 entry, A_3..A_6 of the phase-1 entry
      if (S::VEC && ld == N && lane < 6 && (lane < 2 ? it.slot2 : it.slot1) >= 0 &&
          aligned16(it.ptr[lane < 2 ? 8 + lane : lane]))
        bulk_into(bar, as + lane * N2, it.ptr[lane < 2 ? 8 + lane : lane], N2 * (int)sizeof(T),
                  pol.keep);
      else if (lane < 6 && (lane < 2 ? it.slot2 : it.slot1) >= 0)
      {
        const T *A = static_cast<const T *>(it.ptr[lane < 2 ? 8 + lane : lane]);
        for (int j = 0; j < N; j++)
          for (int i = 0; i < N; i++)
            cp_async<sizeof(T)>(as + lane * N2 + j * N + i, A + i + (long long)j * ld);
      }
      if (it.slot1 < 0)
        return;
      const int h0 = it.idx % K * R, ne = min(R, LH - h0) * LT;
      const T *src = static_cast<const T *>(it.ptr[6]) + (long long)h0 * LT;
      T *buf       = as + S::ASZ;
      if constexpr (S::VEC)
      {
        // a bulk copy per run of chunks between two paddings
        constexpr int RUN = (S::GROUP ? S::GROUP : 1) * N2;
        if (aligned16(src))
          for (int c = lane; c < ne / RUN; c += 32)
            bulk_into(bar, buf + c * (RUN + V), src + c * RUN, RUN * (int)sizeof(T), pol.stream);
        else
          for (int u = lane; u < ne; u += 32)
            cp_async<sizeof(T)>(buf + u + (S::chunk_off(u / N2) - u / N2 * N2), src + u);
      }
      else
      {
        const int sh = (int)((reinterpret_cast<uintptr_t>(src) & 15) / sizeof(T));
        // units [u0, u1) lie whole in the rows; the ends go by elements
        const int u0 = (sh + V - 1) / V, u1 = (sh + ne) / V;
        if (lane == 0)
          bulk_into(bar, buf + u0 * V, src - sh + u0 * V, (u1 - u0) * 16, pol.stream);
        if (lane < u0 * V - sh)
          cp_async<sizeof(T)>(buf + sh + lane, src + lane);
        if (u1 * V + lane < sh + ne)
          cp_async<sizeof(T)>(buf + u1 * V + lane, src + (u1 * V + lane - sh));
      }
    });
    return;
  }

  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::REGS));
  const int gr = warp >> 2, tid = threadIdx.x & 127;
  const Item *items = s_item[gr];
  ControlBars &bars = s_bars[gr];
  for (int i = 0;; ++i)
  {
    const int b    = i & 1;
    const Item &it = items[i % ITEM_SLOTS];
    const bool ok  = __all_sync(0xffffffffu, mbar_wait_bounded(&bars.full[b], (i >> 1) & 1, w.spin));
    if (!ok && lane == 0)
      RingControl<T, K>::leave(w, bars, i, drain);
    const bool go  = ok && it.idx < total;
    const int part = it.idx % K;
    const T *as    = stage_a(gr, b);
    // ---- phase 1, modes 5 and 6 in place
    const int h0   = part * R;
    const int nfib = go && it.slot1 >= 0 ? min(R, LH - h0) * N2 : 0;
    T *xs          = stage_a(gr, b) + S::ASZ;
    if constexpr (!S::VEC)
      if (nfib > 0)
        xs += (reinterpret_cast<uintptr_t>(static_cast<const T *>(it.ptr[6]) +
                                           (long long)h0 * LT) & 15) / sizeof(T);
    if (tid < nfib)
    {
      T *c = xs + S::chunk_off(tid);
      T v[N2];
      load_chunk<T, N>(c, v);
      apply_fast<T, N>(v, as + 5 * N2);
      apply_slow<T, N>(v, as + 4 * N2);
      store_chunk<T, N>(c, v);
    }
    if (!vote_sync<S::G>(gr + 1, go)) // the end of the queue, or a wait that ran out
      return;
    // ---- phase 1, modes 3 and 4; results into W
    if (tid < nfib)
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
    __syncwarp();
    if (lane == 0)
      mbar_arrive(&bars.done[i % ITEM_SLOTS]);
  }
}

// ---------------------------------------------------------------------------
// Tensor-core form (FP64, n = 7 and 8; n = 7 zero padded to 8): head = modes
// 1..3, tail = modes 4..6, everything in mma.sync f64 fragments.  Eight
// computing warps and two control warps.
//   phase 1: a warp takes a head row of n^3 elements, applies the three tail
//   modes (kron8x3_tile) and stores the result into W;
//   phase 2: a block takes 8 columns of W, which lie together (head row after
//   head row).  Warp j_1 loads its (j_2, j_3) x 8 columns, 256 bytes at a time,
//   with the columns on the fragments' G index and applies modes 3 and 2; the results change hands through shared memory
//   (E[j_1][i_2][i_3][c]); warp i_2 applies mode 1 and adds into y.
// E's strides spread the eight columns of four quads over distinct banks for
// both its writes (i_2 = 2t+p) and its reads (j_1 = 2t+p).  A warp's slice of
// E is also its transpose scratch.
template <int N>
struct RingMma
{
  static constexpr int N3 = N * N * N, L = N3 * N3;
  static constexpr int K  = (N3 + 7) / 8;
  static constexpr int WARPS = 8, THREADS = 32 * (WARPS + 2), MINB = 2; // two blocks an SM
  static constexpr int S2 = 66, S1 = 8 * S2 + 2; // strides of E's i_2 and j_1
  static constexpr int ASZ = 6 * N * N;
  static constexpr size_t OFF_E = (2 * (size_t)ASZ * 8 + 15) / 16 * 16;
  // eight head rows, at the offset that their start has in a 16-byte unit
  static constexpr int XLEN     = (8 * N3 + 2) / 2 * 2;
  static constexpr size_t OFF_X = OFF_E + 8 * (size_t)S1 * 8;
  static constexpr size_t SMEM  = OFF_X + 2 * (size_t)XLEN * 8;
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
    kron_ring_mma_kernel(const __grid_constant__ Params p, const __grid_constant__ RingArgs w,
                         long long drain)
{
  using S          = RingMma<N>;
  constexpr int N2 = N * N, N3 = S::N3, K = S::K;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Item s_item[ITEM_SLOTS];
  __shared__ ControlBars s_bars;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double *E     = reinterpret_cast<double *>(smem + S::OFF_E);
  auto stage_a  = [&](int b) { return reinterpret_cast<double *>(smem) + b * S::ASZ; };
  auto stage_x  = [&](int b) { return reinterpret_cast<double *>(smem + S::OFF_X) + b * S::XLEN; };
  const RingPol pol = ring_policies();
  const int total   = (w.nentries + w.lag) * K;
  if (tid == 0)
  {
    control_init(s_bars, S::WARPS);
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == S::WARPS)
  {
    const int ld = p.layout == LAYOUT_XBATCHED ? p.lda : N;
    RingControl<double, K>::run(
        p, w, s_item, s_bars, S::WARPS, lane, drain, [&](const Item &it, int b, uint64_t *bar) {
          double *as = stage_a(b);
          for (int q = lane; q < 6 * N2; q += 32)
          {
            // A_1..A_3 of the phase-2 entry, A_4..A_6 of the phase-1 entry
            const int l = q / N2, ij = q - l * N2, j = ij / N, i = ij - j * N;
            if (l < 3 ? it.slot2 >= 0 : it.slot1 >= 0)
              cp_async<8>(as + q, static_cast<const double *>(it.ptr[l < 3 ? 8 + l : l]) + i +
                                      (long long)j * ld);
          }
          if (it.slot1 < 0)
            return;
          const int h0 = it.idx % K * 8, ne = min(8, N3 - h0) * N3;
          const double *x = static_cast<const double *>(it.ptr[6]) + (long long)h0 * N3;
          double *buf     = stage_x(b);
          const int sh    = aligned16(x) ? 0 : 1;
          const int u1    = (sh + ne) / 2; // units [sh, u1) lie whole in the rows
          if (lane == 0)
            bulk_into(bar, buf + 2 * sh, x - sh + 2 * sh, (u1 - sh) * 16, pol.stream);
          if (sh && lane == 0)
            cp_async<8>(buf + 1, x);
          if (((sh + ne) & 1) && lane == 1)
            cp_async<8>(buf + sh + ne - 1, x + ne - 1);
        });
    return;
  }
  if (warp > S::WARPS)
  {
    if (lane == 0)
      RingControl<double, K>::publish_all(w, &s_item, &s_bars, 1, drain);
    return;
  }

  const int g = lane >> 2, t = lane & 3;
  double *scratch = E + warp * S::S1;
  for (int i = 0;; ++i)
  {
    const int b    = i & 1;
    const Item &it = s_item[i % ITEM_SLOTS];
    const bool ok  = __all_sync(0xffffffffu, mbar_wait_bounded(&s_bars.full[b], (i >> 1) & 1, w.spin));
    if (!ok && lane == 0)
      RingControl<double, K>::leave(w, s_bars, i, drain);
    const bool go    = ok && it.idx < total;
    const int part   = it.idx % K;
    const double *as = stage_a(b);
    // ---- phase 2: this warp's (j_2, j_3) of eight columns, j_1 = warp,
    // columns c = g (on their way during phase 1)
    const int col  = part * 8 + g;
    const bool own = go && it.slot2 >= 0 && warp < N;
    double wv[8][2];
    if (own)
    {
      // j_3 = t + 4 s: four consecutive rows of the tile a load
      const int cw     = min(8, N3 - part * 8);
      const double *wp = static_cast<const double *>(it.ptr[15]) + part * 8 * N3 +
                         (warp * N2 + t) * cw + g;
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
        {
          wv[qq][s] = 0.0;
          if (N == 8 || (qq < N && t + 4 * s < N && g < cw))
            wv[qq][s] = w_load(wp + (qq * N + 4 * s) * cw, pol.keep);
        }
    }
    // ---- phase 1: modes 6, 5, 4 on head row h -> W
    const int h = part * 8 + warp;
    if (go && it.slot1 >= 0 && h < N3)
    {
      AFrag8 f;
      frag_of<N>(f.b1, as + 3 * N2, g, t);
      frag_of<N>(f.b2, as + 4 * N2, g, t);
      frag_of<N>(f.a3, as + 5 * N2, g, t);
      double v[8][2], acc[8][2];
      const bool odd =
          !aligned16(static_cast<const double *>(it.ptr[6]) + (long long)part * 8 * N3);
      const double *row = stage_x(b) + (odd ? 1 : 0) + warp * N3 + g * N + 2 * t;
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
      {
        if (N == 8 && !odd)
        {
          const double2 u = *reinterpret_cast<const double2 *>(row + qq * N2);
          v[qq][0]        = u.x;
          v[qq][1]        = u.y;
        }
        else
#pragma unroll
          for (int s = 0; s < 2; s++)
            v[qq][s] = (N == 8 || (qq < N && g < N && 2 * t + s < N)) ? row[qq * N2 + s] : 0.0;
        acc[qq][0] = acc[qq][1] = 0.0;
      }
      kron8x3_tile<N>(v, acc, f, scratch, g, t);
      // W holds tile after tile of eight columns (n = 7: the last has seven),
      // the head rows of each one after another
      double *wp = static_cast<double *>(it.ptr[7]);
#pragma unroll
      for (int qq = 0; qq < N; qq++)
#pragma unroll
        for (int s = 0; s < 2; s++)
          if (N == 8 || (g < N && 2 * t + s < N))
          {
            const int c  = (2 * t + s) * N2 + qq * N + g;
            const int cw = N == 8 ? 8 : min(8, N3 - (c & ~7));
            w_store(wp + (c & ~7) * N3 + h * cw + (c & 7), acc[qq][s], pol.keep);
          }
    }
    // ---- phase 2, modes 3 and 2
    if (own)
    {
      double b3[2], b2[2], r[8][2];
#pragma unroll
      for (int qq = 0; qq < 8; qq++)
        r[qq][0] = r[qq][1] = 0.0;
#pragma unroll
      for (int s = 0; s < 2; s++)
        b3[s] = (N == 8 || (g < N && t + 4 * s < N)) ? as[2 * N2 + g + (t + 4 * s) * N] : 0.0;
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
    if (!vote_sync<32 * S::WARPS>(1, go)) // the end of the queue, or a wait that ran out
      return;
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
    __syncwarp();
    if (lane == 0)
      mbar_arrive(&s_bars.done[i % ITEM_SLOTS]);
    // E is read by every warp before any warp's next transpose
    asm volatile("bar.sync 1, %0;" ::"n"(32 * S::WARPS) : "memory");
  }
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

// Items that each group has between an entry's phases, and again until its slot
// of W is written anew: a part is published within two items of its being taken
// (1.6: 3% slower at n = 7; 3: 5% slower at n = 8, whose ring then outgrows the
// L2 cache).
constexpr int RING_AHEAD = 2;

template <typename T>
int ring_launch(const void *fn, int threads, int groups, size_t smem, int K, long long L, Params p,
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
  const int ahead        = (int)(RING_AHEAD * blocks * groups / K + 1); // in entries
  w.lag                  = std::max(1, std::min({ahead, w.nentries, w.slots - 1}));
  w.slots                = std::min(w.slots, w.lag + ahead);
  w.magic                = (unsigned)(((1ULL << 32) + w.slots - 1) / w.slots);
  const long long items  = (long long)(w.nentries + w.lag) * K;
  // 32-bit queue positions (one a group taken beyond the end), and the range
  // in which the division by `slots` is exact
  if (items + 3 * blocks > 2147000000LL ||
      ((long long)w.nentries + w.lag) * w.slots >= (1LL << 32))
    return KRON_ERROR_NOT_SUPPORTED;
  ring_init_kernel<T><<<1, 128, 0, stream>>>(w);
  long long drain      = drain_limit();
  const long long grid = std::min(blocks, (items + groups - 1) / groups);
  void *args[]         = {&p, &w, &drain};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(threads), args, smem, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

template <typename T, int N, int R>
int launch_ring_t(const Params &p, const Workspace &wsp, cudaStream_t stream)
{
  using S = RingShape<T, N, R>;
  return ring_launch<T>(reinterpret_cast<const void *>(&kron_ring_kernel<T, N, R>), S::THREADS,
                        S::GROUPS, S::SMEM, S::K, S::L, p, wsp, stream);
}

template <int N>
int launch_ring_mma(const Params &p, const Workspace &wsp, cudaStream_t stream)
{
  using S = RingMma<N>;
  return ring_launch<double>(reinterpret_cast<const void *>(&kron_ring_mma_kernel<N>), S::THREADS,
                             1, S::SMEM, S::K, S::L, p, wsp, stream);
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
    return n == 7   ? launch_ring_t<float, 7, 2>(p, ws, stream)
           : n == 8 ? launch_ring_t<float, 8, 2>(p, ws, stream)
                    : KRON_ERROR_NOT_SUPPORTED;
  return n == 6   ? launch_ring_t<double, 6, 3>(p, ws, stream)
         : n == 7 ? launch_ring_mma<7>(p, ws, stream)
                  : launch_ring_mma<8>(p, ws, stream);
}

} // namespace kron
