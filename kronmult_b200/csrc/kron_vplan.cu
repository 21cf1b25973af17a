// Uneven-batch plans: every entry has its own d and rectangular shapes
// (no reference counterpart; the reference's vbatched needs one launch per
// (d, shape) group, kronmult_vbatched.hpp:17-228, nearly one per entry at
// d >= 3 for random shapes).
//
// kron_vplan_create (host, once) builds a per-entry descriptor table:
//   - Alg. 993 order per entry: forward only when strictly cheaper
//     (kronm.hpp:39-89), and the largest intermediate of that order;
//   - a class by the shared memory the entry needs (two buffers of that
//     intermediate plus its factors) against the per-block budget, half of
//     an SM so that two blocks share each SM: "warp" (<= 512 elements: one
//     warp per entry), "quad" / "half" / "block" (a quarter, a half or all
//     of a block per entry), "huge" (beyond: a two-phase split, head modes
//     [0, q) and tail modes [q, d));
//   - every huge entry is cut into work items: chunk items (phase 1: the
//     tail modes on as many head rows as one block's buffers hold, written
//     to the entry's own region of the workspace) and tile items (phase 2:
//     the head modes on one column tile of that region, added into y);
//   - one queue of huge items, largest entries first, where each entry's
//     tile items follow its chunk items by a lag (a few hundred items, at
//     most ~40 MB of live regions): a tile item waits (bounded) on its
//     entry's chunk counter, which by then is normally complete, and the
//     region it reads is still in L2.
// kron_vplan_execute_async runs one persistent kernel: the huge queue, then
// the block, half, quad and warp classes, each from its own device work
// counter.  All operands reach shared memory by cp.async, so a block keeps
// every byte of its current item in flight at once.  The mode products follow
// a list of steps that the plan computed for each entry (kron_rect.cuh); it
// arrives with the next item's descriptor.
//
// 20000 entries with d in 1..6 and sizes from {2, 3, 4, 6, 8} (0.99 GB): 0.552
// ms, against 0.921 ms when every thread worked out each step's shape and
// divided per fibre (the products were 17 of 29 thousand cycles of a chunk
// item).  Two blocks of 256 threads with factors of up to 36 elements in
// registers are the best split: three blocks (80 registers) 0.616, two of 512
// threads 0.827, one of 512 threads 0.600 ms.  On a non-default
// stream the counter reset and the launch are captured once into a CUDA
// graph and replayed while the operand arrays stay the same.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "kron_launch.h"
#include "kron_ptx.cuh"
#include "kron_rect.cuh"

using namespace kron;

namespace {

constexpr int VP_THREADS = 256;
constexpr int VP_WARPS   = VP_THREADS / 32;
constexpr int VP_AREG    = 36;    // elements of a factor held in registers
constexpr int VP_MINB    = 2;     // blocks per SM the shared-memory budget leaves room for
constexpr int WARP_MAX   = 512;   // elements of the largest intermediate, warp class
constexpr int CLS_WARP = 0, CLS_QUAD = 1, CLS_HALF = 2, CLS_BLOCK = 3, CLS_HUGE = 4;
constexpr int NCLS   = 5;
constexpr int NCOUNT = 8;         // work counters ahead of the per-entry chunk counters

struct VDesc
{
  // fetched as twelve 32-bit words by the kernel's fetch stages
  long long woff;       // huge: element offset of the entry's workspace region
  int k;                // entry index (operands at pA[6k + l], pX[k], pY[k])
  unsigned char d, q, C, pad;  // modes; huge: head modes q, tile columns C
  int nin, nout;        // elements of x and y (huge: of one tail row)
  int hin, hout;        // huge: head rows in and out
  int mi;               // buffer elements: the largest intermediate of the chosen
                        // order (huge: of one chunk of R head rows), and two so
                        // that x may start at an odd element
  int mi2;              // huge: phase-2 buffer elements (tile rows x C)
  int R;                // huge: head rows per chunk item
  int nchunk;           // huge: chunk items (its tile items wait for all)
};

static_assert(sizeof(VDesc) == 48, "VDesc is fetched as 12 words");

// an entry's mode products (huge: the d - q tail steps, then the q head steps)
struct VSteps
{
  RectStep st[MAXD];
};
constexpr int VSTEP_WORDS = sizeof(VSteps) / 4;
static_assert(VSTEP_WORDS <= 32, "fetched as a word a lane");

// kind 0: chunk item, head rows [lo, hi); kind 1: tile item, column tile lo
// of the huge entry desc[e]
struct VItem
{
  int e, lo, hi, kind;
};

struct VParams
{
  const VDesc *desc;          // [huge | block | half | quad | warp]
  const VSteps *steps;        // the same order
  const VItem *items;         // the huge queue
  int nhuge, nblock, nhalf, nquad, nwarp;
  int nitems;
  int *counters;              // [0] huge queue, [1] block, [2] warp, [4] half,
                              // [5] quad; [NCOUNT + i] chunks done of huge entry i
  int *status;                // the library's device status word
  long long spin;             // polls before a chunk wait gives up
  const double *const *pA;
  const double *const *pX;
  double *const *pY;
  double *ws;                 // huge class: per-entry regions
  int budget;                 // shared elements per block, BUF_SLACK among them
};

// 8-byte global -> shared copy through the LSU's asynchronous path
// (zero-filled when !valid; src must still point into the operand).
__device__ __forceinline__ void cp8(double *dst, const double *src, bool valid = true)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(ptx::smem_addr(dst)),
               "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}

__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ int ld_acquire(const int *p)
{
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The steps' factors (leading dimension m_l: each contiguous) into As in step
// order, a warp a step.
__device__ __forceinline__ void vp_load_factors(const RectStep *st, int ns, double *As,
                                                const double *const *A, int t, int GS)
{
  const int warp = t >> 5, lane = t & 31, nw = GS >> 5;
  int o = 0;
  for (int s = 0; s < ns; s++)
  {
    const int sz = st[s].nq * st[s].mq;
    if (s % nw == warp)
    {
      const double *a = A[st[s].mode];
      for (int u = lane; u < sz; u += 32)
        cp8(As + o + u, a + u);
    }
    o += sz;
  }
}

// `count` elements at src to buf + the offset src has in its 16-byte unit,
// 16 bytes at a time but for the ends; returns where they start.
__device__ __forceinline__ double *vp_load_x(double *buf, const double *src, int count, int t,
                                             int GS)
{
  const int sh = (int)((reinterpret_cast<uintptr_t>(src) >> 3) & 1);
  const int u1 = (sh + count) / 2; // units [sh, u1) lie whole in the source
  for (int u = sh + t; u < u1; u += GS)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_addr(buf + 2 * u)),
                 "l"(src - sh + 2 * u)
                 : "memory");
  if (sh && t == 0)
    cp8(buf + 1, src);
  if (((sh + count) & 1) && t == GS - 1)
    cp8(buf + sh + count - 1, src + count - 1);
  return buf + sh;
}

// rows consecutive vectors (x contiguous) computed by a group of GS threads
// in buffers b0 / b1 (each >= rows x the largest intermediate and two),
// factors at As; the results go to out (contiguous): added into y, or stored
// into the workspace region.  hook(s) runs the next item's fetch stage s at
// four points: after the copies are issued, after they land, before the
// results go out, and before the closing barrier.
template <bool STORE, typename Hook>
__device__ __forceinline__ void vp_run(const RectStep *st, int ns, int rows, int nin, int nout,
                                       const double *x, double *out, double *b0, double *b1,
                                       double *As, const double *const *A, int t, int GS, int g,
                                       const Hook &hook)
{
  vp_load_factors(st, ns, As, A, t, GS);
  double *cur = vp_load_x(b0, x, rows * nin, t, GS), *nxt = b1;
  hook(1);
  cp_wait_all();
  group_sync(g, GS);
  hook(2);
  rect_modes<double, VP_AREG>(st, ns, rows, cur, nxt, As, t, GS, g);
  hook(3);
  const int count = rows * nout;
  if constexpr (STORE)
  {
    if (ptx::aligned16(cur) && ptx::aligned16(out))
    {
      for (int i = t; i < count / 2; i += GS)
        reinterpret_cast<double2 *>(out)[i] = reinterpret_cast<const double2 *>(cur)[i];
      if ((count & 1) && t == 0)
        out[count - 1] = cur[count - 1];
    }
    else
      for (int i = t; i < count; i += GS)
        out[i] = cur[i];
  }
  else
    for (int i = t; i < count; i += GS)
      red_add(out + i, cur[i]);
  hook(4);
  group_sync(g, GS);
}

// One column tile of a huge entry's region: rin rows of C columns at stride
// in_row (the first Cc valid, the rest zero-filled), the head modes, and
// the Cc valid columns added into y (rout rows, row stride out_row).  Whole
// block; hook as for vp_run.
template <typename Hook>
__device__ __forceinline__ void vp_run_tile(const RectStep *st, int ns, int rin, int rout,
                                            const double *w, int in_row, int C, int Cc, double *y,
                                            int out_row, double *b0, double *b1, double *As,
                                            const double *const *A, int tid, const Hook &hook)
{
  vp_load_factors(st, ns, As, A, tid, VP_THREADS);
  const int lane = tid & 31, warp = tid >> 5;
  if (((C | Cc | in_row) & 1) == 0 && ptx::aligned16(w))
  {
    for (int h = warp; h < rin; h += VP_WARPS)
      for (int c = 2 * lane; c < C; c += 64)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_addr(b0 + h * C + c)),
                     "l"(w + (long long)h * in_row + (c < Cc ? c : 0)), "r"(c < Cc ? 16 : 0)
                     : "memory");
  }
  else
    for (int h = warp; h < rin; h += VP_WARPS)
      for (int c = lane; c < C; c += 32)
        cp8(b0 + h * C + c, w + (long long)h * in_row + (c < Cc ? c : 0), c < Cc);
  hook(1);
  cp_wait_all();
  __syncthreads();
  hook(2);
  double *cur = b0, *nxt = b1;
  rect_modes<double, VP_AREG>(st, ns, 1, cur, nxt, As, tid, VP_THREADS, 0);
  hook(3);
  for (int i = warp; i < rout; i += VP_WARPS)
    for (int c = lane; c < Cc; c += 32)
      red_add(y + (long long)i * out_row + c, cur[i * C + c]);
  hook(4);
  __syncthreads();
}

// What a group needs to start its next item, in shared memory.  The
// group's first warp fetches it in stages during the current item, one
// dependent load per stage (queue index, item, descriptor, operand
// pointers), so none of those round trips stalls the group.
struct NextSlot
{
  int idx;               // queue / list position (>= the count: no more work)
  int ready;             // huge tile item: its entry's chunks were complete
  VItem it;              // huge queue only
  VDesc e;
  VSteps s;
  const double *ptr[8];  // A_1..A_6, x, y
};

// The fetching warp's registers between stages.
struct Fetch
{
  int r;                 // lane 0: the counter's old value; lanes: a word in flight
  int w;                 // lanes: a word of the steps in flight
  int nidx;
  const double *p;       // lanes 0-7: a pointer in flight
};

// Stages of the fetch for the huge queue (kind = true) or a class list.
// Stage 0 takes the next position; 1 loads the item (huge) or the
// descriptor; 2 stores it and loads the descriptor (huge) or the pointers;
// 3 and 4 finish.  Every store to the slot happens after the current item
// has read the slot (the first barrier of the item lies between).
template <bool HUGE>
__device__ __forceinline__ void fetch_stage(int s, Fetch &f, NextSlot &slot, const VParams &vp,
                                            const VDesc *list, int n, int *counter, int lane)
{
  const unsigned FULL = 0xffffffffu;
  if (s == 0)
  {
    if (lane == 0)
      f.r = atomicAdd(counter, 1);
    return;
  }
  if (s == 1)
  {
    f.nidx = __shfl_sync(FULL, f.r, 0);
    if (f.nidx < n)
    {
      if (HUGE && lane < 4)
        f.r = reinterpret_cast<const int *>(vp.items + f.nidx)[lane];
      if (!HUGE && lane < 12)
        f.r = reinterpret_cast<const int *>(list + f.nidx)[lane];
      if (!HUGE && lane < VSTEP_WORDS)
        f.w = reinterpret_cast<const int *>(vp.steps + (list - vp.desc) + f.nidx)[lane];
    }
    return;
  }
  const bool more = f.nidx < n;
  if (HUGE)
  {
    if (s == 2)
    {
      if (lane == 0)
        slot.idx = f.nidx;
      if (more && lane < 4)
        reinterpret_cast<int *>(&slot.it)[lane] = f.r;
      __syncwarp();
      if (more && lane < 12)
        f.r = reinterpret_cast<const int *>(vp.desc + slot.it.e)[lane];
      if (more && lane < VSTEP_WORDS)
        f.w = reinterpret_cast<const int *>(vp.steps + slot.it.e)[lane];
    }
    else if (s == 3)
    {
      if (more && lane < 12)
        reinterpret_cast<int *>(&slot.e)[lane] = f.r;
      if (more && lane < VSTEP_WORDS)
        reinterpret_cast<int *>(&slot.s)[lane] = f.w;
      __syncwarp();
      if (more && lane < 8)
      {
        const int k = slot.e.k, d = slot.e.d;
        f.p = lane < 6 ? (lane < d ? vp.pA[6LL * k + lane] : nullptr)
                       : (lane == 6 ? vp.pX[k] : vp.pY[k]);
      }
      if (more && lane == 8)
        f.r = slot.it.kind == 1 && ld_acquire(vp.counters + NCOUNT + slot.it.e) >= slot.e.nchunk;
    }
    else
    {
      if (more && lane < 8)
        slot.ptr[lane] = f.p;
      if (more && lane == 8)
        slot.ready = f.r;
    }
  }
  else
  {
    if (s == 2)
    {
      if (lane == 0)
        slot.idx = f.nidx;
      if (more && lane < 12)
        reinterpret_cast<int *>(&slot.e)[lane] = f.r;
      if (more && lane < VSTEP_WORDS)
        reinterpret_cast<int *>(&slot.s)[lane] = f.w;
      __syncwarp();
      if (more && lane < 8)
      {
        const int k = slot.e.k, d = slot.e.d;
        f.p = lane < 6 ? (lane < d ? vp.pA[6LL * k + lane] : nullptr)
                       : (lane == 6 ? vp.pX[k] : vp.pY[k]);
      }
    }
    else if (s == 3)
    {
      if (more && lane < 8)
        slot.ptr[lane] = f.p;
    }
  }
}

// Thread 0 polls the entry's chunk counter (acquire) until `need` chunk
// items are done, at most `spin` polls; on giving up it records 1 in the
// status word.  Returns the outcome to the whole block.
__device__ __forceinline__ bool vp_wait_chunks(const VParams &vp, int e, int need, int *s_flag,
                                               int tid)
{
  if (tid == 0)
  {
    const int *done = vp.counters + NCOUNT + e;
    int ok          = 1;
    long long polls = 0;
    while (ld_acquire(done) < need)
    {
      if (++polls > vp.spin)
      {
        ok = 0;
        if (vp.status)
          atomicExch(vp.status, 1);
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    *s_flag = ok;
  }
  __syncthreads();
  return *s_flag != 0;
}

// Entries of one class run by groups of GS threads, VP_THREADS / GS per
// block, each group with its own slice of shared memory, barrier and slots
// (the current item's and the next one's).
template <int GS>
__device__ __forceinline__ void group_class(const VParams &vp, const VDesc *list, int n,
                                            int *counter, double *smem, NextSlot (*slots)[2],
                                            int tid)
{
  constexpr int NG = VP_THREADS / GS;
  const int g = tid / GS, t = tid - (tid / GS) * GS, lane = tid & 31;
  double *b0    = smem + (long long)g * ((vp.budget / NG) & ~1);
  const bool fw = t < 32; // the group's first warp fetches
  Fetch f{0, 0, 0, nullptr};
  if (fw)
    for (int st = 0; st < 4; st++)
    {
      fetch_stage<false>(st, f, slots[g][0], vp, list, n, counter, lane);
      __syncwarp();
    }
  group_sync(g, GS);
  for (int b = 0;; b ^= 1)
  {
    const NextSlot &slot = slots[g][b];
    NextSlot &next       = slots[g][b ^ 1];
    if (slot.idx >= n)
      break;
    if (fw)
      fetch_stage<false>(0, f, next, vp, list, n, counter, lane);
    const VDesc &e = slot.e;
    vp_run<false>(slot.s.st, e.d, 1, e.nin, e.nout, slot.ptr[6],
                  const_cast<double *>(slot.ptr[7]), b0, b0 + e.mi, b0 + 2 * e.mi, slot.ptr, t,
                  GS, g, [&](int st) {
                    if (fw && st < 4)
                      fetch_stage<false>(st, f, next, vp, list, n, counter, lane);
                  });
  }
  __syncthreads(); // the next class lays its slices (and slots) over these
}

// The huge queue, then the block, half, quad and warp classes.
__global__ void __launch_bounds__(VP_THREADS, VP_MINB)
    kron_vplan_kernel(const __grid_constant__ VParams vp)
{
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_flag;
  __shared__ NextSlot s_slot[VP_WARPS][2];
  const int tid = threadIdx.x, lane = tid & 31;
  const bool fw = tid < 32;
  bool dead = false; // a chunk wait of this block gave up: skip later tile items

  Fetch f{0, 0, 0, nullptr};
  if (fw)
    for (int st = 0; st < 5; st++)
    {
      fetch_stage<true>(st, f, s_slot[0][0], vp, nullptr, vp.nitems, &vp.counters[0], lane);
      __syncwarp();
    }
  __syncthreads();
  for (int b = 0;; b ^= 1)
  {
    const NextSlot &slot = s_slot[0][b];
    NextSlot &next       = s_slot[0][b ^ 1];
    if (slot.idx >= vp.nitems)
      break;
    auto hook = [&](int st) {
      if (fw)
        fetch_stage<true>(st, f, next, vp, nullptr, vp.nitems, &vp.counters[0], lane);
    };
    hook(0);
    const VItem &it = slot.it;
    const VDesc &e  = slot.e;
    double *wr      = vp.ws + e.woff;
    if (it.kind == 0)
    {
      // phase 1: tail modes on head rows [lo, hi) -> the entry's region
      vp_run<true>(slot.s.st, e.d - e.q, it.hi - it.lo, e.nin, e.nout,
                   slot.ptr[6] + (long long)it.lo * e.nin, wr + (long long)it.lo * e.nout, smem,
                   smem + e.mi, smem + 2 * e.mi, slot.ptr, tid, VP_THREADS, 0, hook);
      // vp_run ended with a block barrier: every store of the chunk is issued
      if (tid == 0)
      {
        __threadfence();
        atomicAdd(vp.counters + NCOUNT + it.e, 1);
      }
    }
    else
    {
      // phase 2: head modes on column tile lo of the region -> y
      if (!slot.ready && !dead && !vp_wait_chunks(vp, it.e, e.nchunk, &s_flag, tid))
        dead = true;
      if (dead)
      {
        // keep the fetch going: the stages still run, the tile does not
        for (int st = 1; st < 5; st++)
        {
          hook(st);
          __syncthreads();
        }
        continue;
      }
      const int c0 = it.lo * e.C;
      vp_run_tile(slot.s.st + (e.d - e.q), e.q, e.hin, e.hout, wr + c0, e.nout, e.C,
                  min((int)e.C, e.nout - c0), const_cast<double *>(slot.ptr[7]) + c0, e.nout,
                  smem, smem + e.mi2, smem + 2 * e.mi2, slot.ptr, tid, hook);
    }
  }
  __syncthreads();

  const VDesc *blk = vp.desc + vp.nhuge;
  group_class<VP_THREADS>(vp, blk, vp.nblock, &vp.counters[1], smem, s_slot, tid);
  blk += vp.nblock;
  group_class<VP_THREADS / 2>(vp, blk, vp.nhalf, &vp.counters[4], smem, s_slot, tid);
  blk += vp.nhalf;
  group_class<VP_THREADS / 4>(vp, blk, vp.nquad, &vp.counters[5], smem, s_slot, tid);
  blk += vp.nquad;
  group_class<32>(vp, blk, vp.nwarp, &vp.counters[2], smem, s_slot, tid);
}

} // namespace

struct kron_vplan_st
{
  int batch;
  int nhuge, nblock, nhalf, nquad, nwarp;
  int nitems;
  VDesc *d_desc;
  VSteps *d_steps;            // in d_desc's block
  VItem *d_items;
  int *d_counters;            // NCOUNT work counters + one chunk counter per huge entry
  double flops;
  size_t ws_bytes;
  int budget;                 // shared elements per block, BUF_SLACK among them
  int grid_work;              // work units of the launch (grid upper bound)
  // graph cache
  cudaGraphExec_t exec;
  const void *gA, *gX, *gY, *gW;
  size_t gWcap;
};

namespace {

long long even(long long v) { return (v + 1) & ~1LL; }

// Alg. 993 order of an entry (forward only when strictly cheaper,
// kronm.hpp:83-89), its flops and its largest intermediate, in one walk each
// way.
struct OrderCost
{
  bool forward;
  double flops;
  long long elems;
};

OrderCost order_cost(int d, const int *m, const int *n)
{
  // products of the sizes before and from each mode on
  long long pm[MAXD + 1], pn[MAXD + 1], sm[MAXD + 1], sn[MAXD + 1];
  pm[0] = pn[0] = sm[d] = sn[d] = 1;
  for (int l = 0; l < d; l++)
  {
    pm[l + 1]     = pm[l] * m[l];
    pn[l + 1]     = pn[l] * n[l];
    sm[d - 1 - l] = sm[d - l] * m[d - 1 - l];
    sn[d - 1 - l] = sn[d - l] * n[d - 1 - l];
  }
  long long fmax = pn[d], bmax = pn[d];
  double ff = 0.0, fb = 0.0;
  for (int l = 0; l < d; l++)
  {
    ff += 2.0 * (double)(pm[l + 1] * sn[l]);
    fmax = std::max(fmax, pm[l + 1] * sn[l + 1]);
    fb += 2.0 * (double)(pn[l + 1] * sm[l]);
    bmax = std::max(bmax, pn[l] * sm[l]);
  }
  return ff < fb ? OrderCost{true, ff, fmax} : OrderCost{false, fb, bmax};
}

// Entries by falling cost, equal ones in entry order: a counting sort on the
// bits of the (positive) cost as a float.
struct Ranked
{
  float cost;
  int k;
};

void sort_by_cost(std::vector<Ranked> &v)
{
  std::vector<Ranked> tmp(v.size());
  for (int shift = 0; shift < 33; shift += 11)
  {
    unsigned count[2049] = {};
    auto key = [&](const Ranked &r) {
      unsigned b;
      std::memcpy(&b, &r.cost, 4);
      return (~b >> shift) & 2047u;
    };
    for (const Ranked &r : v)
      count[key(r) + 1]++;
    for (int i = 0; i < 2048; i++)
      count[i + 1] += count[i];
    for (const Ranked &r : v)
      tmp[count[key(r)]++] = r;
    v.swap(tmp);
  }
}

// Elements beyond an entry's budget that its buffers may take: two a buffer,
// where x starts at the offset it has in a 16-byte unit, and a chunk's odd rows.
constexpr int BUF_SLACK = 6;

// Two-phase split of a huge entry for a block of `budget` shared elements:
// phase 1 applies modes [q, d) to chunks of R head rows, phase 2 modes
// [0, q) to column tiles of C columns.  Prefers tiles of >= 16 columns
// (128-byte row segments), then the smallest region (Nhead x Mtail).
struct HugeSplit
{
  int q, C, R, fwd1, fwd2;
  long long mi1, mi2; // buffer elements: per head row (phase 1), per column (phase 2)
};

bool plan_huge(int d, const int *m, const int *n, long long budget, HugeSplit &best)
{
  bool found = false;
  long long best_w = 0;
  int best_c = 0;
  for (int q = 1; q < d; q++)
  {
    const OrderCost o1 = order_cost(d - q, m + q, n + q);
    const OrderCost o2 = order_cost(q, m, n);
    const long long r1 = o1.elems, r2 = o2.elems;
    long long a1 = 0, a2 = 0, Nhead = 1, Mtail = 1;
    for (int l = 0; l < q; l++)
    {
      a2 += (long long)m[l] * n[l];
      Nhead *= n[l];
    }
    for (int l = q; l < d; l++)
    {
      a1 += (long long)m[l] * n[l];
      Mtail *= m[l];
    }
    const long long R = (budget - even(a1) - 2) / (2 * r1);
    const long long C = std::min<long long>({255, Mtail, (budget - even(a2) - 2) / (2 * r2)});
    if (R < 1 || C < 1)
      continue;
    const int cq        = (int)std::min<long long>(C, 16);
    const long long wsz = Nhead * Mtail;
    if (!found || cq > best_c || (cq == best_c && wsz < best_w))
    {
      best = HugeSplit{q, (int)C, (int)std::min<long long>(R, 65535), o1.forward ? 1 : 0,
                       o2.forward ? 1 : 0, r1, r2};
      best_c = cq;
      best_w = wsz;
      found  = true;
    }
  }
  return found;
}

} // namespace

extern "C" int kron_vplan_create(kron_vplan_t *plan, int batchCount, int const shapes[])
{
  if (!plan || batchCount < 0 || (batchCount > 0 && !shapes))
    return KRON_ERROR_INVALID_VALUE;
  *plan = nullptr;
  const DeviceInfo &di = device_info();
  // shared elements per block: two blocks per SM (1 KB of each block's share
  // is reserved by the hardware; 4 KB cover the kernel's own variables and the
  // slack).  A plan with a shape that only 2 KB more can hold (a factor of 118 x
  // 118) runs one block per SM.
  const long long two_blocks =
      (std::min<long long>(di.max_smem_optin, di.smem_per_sm / VP_MINB - 1024) - 4096) / 8 & ~1LL;
  static_assert(sizeof(NextSlot) * 2 * VP_WARPS + 8 * BUF_SLACK + 64 <= 4096,
                "the kernel's own variables");
  long long budget = two_blocks;
  // class and cost of every entry, then descriptors and steps in queue order
  std::vector<Ranked> cls[NCLS];
  std::vector<HugeSplit> splits; // of the huge entries, in entry order
  std::vector<int> split_of(batchCount, -1);
  double total_flops = 0.0;
  int m[MAXD], n[MAXD];
  auto shape_of = [&](int k) {
    const int *s = shapes + 13LL * k;
    for (int l = 0; l < s[0]; l++)
    {
      m[l] = s[1 + 2 * l];
      n[l] = s[2 + 2 * l];
    }
    return s[0];
  };
  auto classify = [&]() {
    for (int k = 0; k < batchCount; k++)
    {
      const int d = shapes[13LL * k];
      if (d < 1 || d > MAXD)
        return (int)KRON_ERROR_INVALID_VALUE;
      shape_of(k);
      long long asz = 0;
      for (int l = 0; l < d; l++)
      {
        if (m[l] < 1 || n[l] < 1 || m[l] > 255 || n[l] > 255)
          return (int)KRON_ERROR_INVALID_VALUE;
        asz += (long long)m[l] * n[l];
      }
      const OrderCost oc = order_cost(d, m, n);
      total_flops += oc.flops;
      const long long mi   = even(oc.elems) + 2;
      const long long need = 2 * mi + even(asz);
      int c;
      if (mi <= WARP_MAX && need <= (budget / VP_WARPS & ~1LL))
        c = CLS_WARP;
      else if (need <= (budget / 4 & ~1LL))
        c = CLS_QUAD;
      else if (need <= (budget / 2 & ~1LL))
        c = CLS_HALF;
      else if (need <= budget + 4) // with the four elements of x's offsets
        c = CLS_BLOCK;
      else
      {
        c = CLS_HUGE;
        HugeSplit hs;
        if (!plan_huge(d, m, n, budget, hs))
          return (int)KRON_ERROR_NOT_SUPPORTED;
        split_of[k] = (int)splits.size();
        splits.push_back(hs);
      }
      cls[c].push_back(Ranked{(float)oc.flops, k});
    }
    return (int)KRON_SUCCESS;
  };
  int rc = classify();
  if (rc == KRON_ERROR_NOT_SUPPORTED)
  {
    budget = two_blocks + 256;
    for (auto &c : cls)
      c.clear();
    splits.clear();
    total_flops = 0.0;
    rc          = classify();
  }
  if (rc != KRON_SUCCESS)
    return rc;
  kron_vplan_st *pl = new (std::nothrow) kron_vplan_st();
  if (!pl)
    return KRON_ERROR_ALLOC;
  // descriptors, then steps: one device block
  const size_t desc_bytes = (sizeof(VDesc) * batchCount + 15) / 16 * 16;
  std::vector<unsigned char> host(desc_bytes + sizeof(VSteps) * batchCount);
  VDesc *all    = reinterpret_cast<VDesc *>(host.data());
  VSteps *steps = reinterpret_cast<VSteps *>(host.data() + desc_bytes);
  int at        = 0;
  for (int c : {CLS_HUGE, CLS_BLOCK, CLS_HALF, CLS_QUAD, CLS_WARP})
  {
    sort_by_cost(cls[c]);
    for (const Ranked &r : cls[c])
    {
      VDesc &e     = all[at];
      RectStep *st = steps[at].st;
      at++;
      const int d = shape_of(r.k);
      e.k         = r.k;
      e.d         = (unsigned char)d;
      e.nin = e.nout = e.hin = e.hout = 1;
      if (c != CLS_HUGE)
      {
        for (int l = 0; l < d; l++)
        {
          e.nin *= n[l];
          e.nout *= m[l];
        }
        const OrderCost oc = order_cost(d, m, n);
        // two more: x starts at the offset it has in a 16-byte unit
        e.mi = (int)even(oc.elems) + 2;
        rect_plan(st, d, m, n, 0, oc.forward, 1);
        continue;
      }
      const HugeSplit &hs = splits[split_of[r.k]];
      e.q = (unsigned char)hs.q;
      e.C = (unsigned char)hs.C;
      for (int l = 0; l < d; l++)
      {
        (l < hs.q ? e.hin : e.nin) *= n[l];
        (l < hs.q ? e.hout : e.nout) *= m[l];
      }
      rect_plan(st, d - hs.q, m + hs.q, n + hs.q, hs.q, hs.fwd1 != 0, 1);
      rect_plan(st + (d - hs.q), hs.q, m, n, 0, hs.fwd2 != 0, hs.C);
      // chunks of equal size, at most R rows each
      const long long nchunk = (e.hin + hs.R - 1) / hs.R;
      const long long R      = (e.hin + nchunk - 1) / nchunk;
      e.R      = (int)R;
      e.nchunk = (int)nchunk;
      e.mi     = (int)even(R * hs.mi1) + 2;
      e.mi2    = (int)even(hs.C * hs.mi2);
    }
  }
  pl->batch  = batchCount;
  pl->nhuge  = (int)cls[CLS_HUGE].size();
  pl->nblock = (int)cls[CLS_BLOCK].size();
  pl->nhalf  = (int)cls[CLS_HALF].size();
  pl->nquad  = (int)cls[CLS_QUAD].size();
  pl->nwarp  = (int)cls[CLS_WARP].size();

  // The huge queue: entries largest first; an entry's tile items enter the
  // queue once `lag_items` items or `lag_elems` elements of live regions
  // separate them from its chunk items (whichever comes first), so a tile
  // item rarely waits and its region is still in L2.  Regions start on
  // 128-byte boundaries.
  std::vector<VItem> items;
  const long long lag_items = 2LL * di.sms * VP_MINB;
  const long long lag_elems = 40LL << 17; // 40 MB of regions
  struct Pending
  {
    int e;
    size_t pos;
    long long elems;
  };
  std::vector<Pending> pend;
  size_t pend_head   = 0;
  long long live     = 0;
  long long woff     = 0;
  auto emit_tiles = [&](const Pending &p) {
    const VDesc &e     = all[p.e];
    const long long nt = (e.nout + e.C - 1) / e.C;
    for (long long t = 0; t < nt; t++)
      items.push_back(VItem{p.e, (int)t, (int)t + 1, 1});
    live -= p.elems;
  };
  for (int i = 0; i < pl->nhuge; i++)
  {
    VDesc &e = all[i];
    e.woff   = woff;
    const long long Nhead = e.hin, Mtail = e.nout;
    const long long region = (Nhead * Mtail + 15) & ~15LL;
    woff += region;
    for (long long h0 = 0; h0 < Nhead; h0 += e.R)
      items.push_back(VItem{i, (int)h0, (int)std::min<long long>(Nhead, h0 + e.R), 0});
    pend.push_back(Pending{i, items.size(), region});
    live += region;
    while (pend_head < pend.size() &&
           ((long long)(items.size() - pend[pend_head].pos) >= lag_items || live > lag_elems))
      emit_tiles(pend[pend_head++]);
  }
  while (pend_head < pend.size())
    emit_tiles(pend[pend_head++]);

  pl->nitems     = (int)items.size();
  pl->flops      = total_flops;
  pl->budget     = (int)budget + BUF_SLACK;
  pl->ws_bytes   = (size_t)woff * 8;
  pl->grid_work  = (int)std::min<long long>(
      1LL << 30, (long long)items.size() + pl->nblock + (pl->nhalf + 1) / 2 +
                     (pl->nquad + 3) / 4 + (pl->nwarp + VP_WARPS - 1) / VP_WARPS);
  pl->exec       = nullptr;
  pl->d_desc     = nullptr;
  pl->d_items    = nullptr;
  pl->d_counters = nullptr;
  const size_t ncount = NCOUNT + (size_t)pl->nhuge;
  if (kron::dev_malloc((void **)&pl->d_counters, ncount * sizeof(int)) != cudaSuccess ||
      (batchCount > 0 && kron::dev_malloc((void **)&pl->d_desc, host.size()) != cudaSuccess) ||
      (!items.empty() && kron::dev_malloc((void **)&pl->d_items, sizeof(VItem) * items.size()) != cudaSuccess))
  {
    kron::dev_free(pl->d_items);
    kron::dev_free(pl->d_desc);
    kron::dev_free(pl->d_counters);
    delete pl;
    return KRON_ERROR_ALLOC;
  }
  pl->d_steps = reinterpret_cast<VSteps *>(reinterpret_cast<unsigned char *>(pl->d_desc) + desc_bytes);
  if ((batchCount > 0 && cudaMemcpy(pl->d_desc, host.data(), host.size(),
                                    cudaMemcpyHostToDevice) != cudaSuccess) ||
      (!items.empty() && cudaMemcpy(pl->d_items, items.data(), sizeof(VItem) * items.size(),
                                    cudaMemcpyHostToDevice) != cudaSuccess))
  {
    kron::dev_free(pl->d_items);
    kron::dev_free(pl->d_desc);
    kron::dev_free(pl->d_counters);
    delete pl;
    return KRON_ERROR_LAUNCH;
  }
  *plan = pl;
  return KRON_SUCCESS;
}

extern "C" int kron_vplan_destroy(kron_vplan_t plan)
{
  if (!plan)
    return KRON_SUCCESS;
  if (plan->exec)
    cudaGraphExecDestroy(plan->exec);
  kron::dev_free(plan->d_items);
  kron::dev_free(plan->d_desc);
  kron::dev_free(plan->d_counters);
  delete plan;
  return KRON_SUCCESS;
}

extern "C" size_t kron_vplan_workspace_bytes(kron_vplan_t plan) { return plan ? plan->ws_bytes : 0; }
extern "C" double kron_vplan_flops(kron_vplan_t plan) { return plan ? plan->flops : 0.0; }

static int vplan_launch_all(kron_vplan_t pl, double const *const *A, double **X, double **Y,
                            void *W, cudaStream_t s)
{
  if (cudaMemsetAsync(pl->d_counters, 0, (NCOUNT + (size_t)pl->nhuge) * sizeof(int), s) !=
      cudaSuccess)
    return KRON_ERROR_LAUNCH;
  if (pl->grid_work <= 0)
    return KRON_SUCCESS;
  VParams vp;
  std::memset(&vp, 0, sizeof(vp));
  vp.desc     = pl->d_desc;
  vp.steps    = pl->d_steps;
  vp.items    = pl->d_items;
  vp.nhuge    = pl->nhuge;
  vp.nblock   = pl->nblock;
  vp.nhalf    = pl->nhalf;
  vp.nquad    = pl->nquad;
  vp.nwarp    = pl->nwarp;
  vp.nitems   = pl->nitems;
  vp.counters = pl->d_counters;
  vp.status   = device_status_ptr();
  vp.spin     = wait_limit();
  vp.pA       = A;
  vp.pX       = X;
  vp.pY       = Y;
  vp.ws       = static_cast<double *>(W);
  vp.budget   = pl->budget;
  void *args[]      = {&vp};
  const void *fm    = reinterpret_cast<const void *>(&kron_vplan_kernel);
  const size_t smem = (size_t)pl->budget * 8;
  int occ           = 1;
  if (cached_occupancy(fm, VP_THREADS, smem, &occ) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  // persistent: every block stays resident until the queues run dry
  const int grid =
      (int)std::max<long long>(1, std::min<long long>((long long)device_info().sms * occ,
                                                      pl->grid_work));
  if (cudaLaunchKernel(fm, dim3(grid), dim3(VP_THREADS), args, smem, s) != cudaSuccess)
    return KRON_ERROR_LAUNCH;
  return KRON_SUCCESS;
}
extern "C" int kron_vplan_execute_async(kron_vplan_t plan, double const *const Aarray_[],
                                        double *pX_[], double *pY_[], void *W,
                                        size_t Wcapacity_bytes, kron_stream_t stream)
{
  if (!plan)
    return KRON_ERROR_INVALID_VALUE;
  if (plan->batch == 0)
    return KRON_SUCCESS;
  if (!Aarray_ || !pX_ || !pY_)
    return KRON_ERROR_INVALID_VALUE;
  cudaStream_t s = (cudaStream_t)stream;
  if (plan->ws_bytes > 0 && (!W || Wcapacity_bytes < plan->ws_bytes))
    return KRON_ERROR_WORKSPACE;

  // Graphs only on explicit streams that are not already capturing.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  bool use_graph             = (s != nullptr) && cudaStreamIsCapturing(s, &cs) == cudaSuccess &&
                   cs == cudaStreamCaptureStatusNone;
  if (!use_graph)
  {
    int rc = vplan_launch_all(plan, Aarray_, pX_, pY_, W, s);
    if (rc != KRON_SUCCESS)
      return rc;
    return cudaGetLastError() == cudaSuccess ? KRON_SUCCESS : KRON_ERROR_LAUNCH;
  }
  const bool same = plan->exec && plan->gA == Aarray_ && plan->gX == pX_ && plan->gY == pY_ &&
                    plan->gW == W && plan->gWcap == Wcapacity_bytes;
  if (!same)
  {
    if (plan->exec)
    {
      cudaGraphExecDestroy(plan->exec);
      plan->exec = nullptr;
    }
    // kernel attributes are set outside the capture
    int rc = vplan_launch_all(plan, Aarray_, pX_, pY_, W, s);
    if (rc != KRON_SUCCESS)
      return rc;
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
      return KRON_ERROR_LAUNCH;
    rc             = vplan_launch_all(plan, Aarray_, pX_, pY_, W, s);
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (rc != KRON_SUCCESS)
    {
      if (graph)
        cudaGraphDestroy(graph);
      return rc;
    }
    if (ce != cudaSuccess || !graph)
      return KRON_ERROR_LAUNCH;
    cudaGraphExec_t exec = nullptr;
    ce                   = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess)
      return KRON_ERROR_LAUNCH;
    plan->exec  = exec;
    plan->gA    = Aarray_;
    plan->gX    = pX_;
    plan->gY    = pY_;
    plan->gW    = W;
    plan->gWcap = Wcapacity_bytes;
    return KRON_SUCCESS; // this execution ran directly above
  }
  return cudaGraphLaunch(plan->exec, s) == cudaSuccess ? KRON_SUCCESS : KRON_ERROR_LAUNCH;
}
