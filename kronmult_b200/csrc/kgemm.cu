// Batched small GEMM:  C_k = alpha op(A_k) op(B_k) + beta C_k
// Replaces kgemm_{nn,nt,tt}_batched (kgemm_nn_batched.hpp:7-58 and the
// device GEMMs kgemm_nn.hpp:12-203, kgemm_nt.hpp:10-202, kgemm_tt.hpp:10-200).
//
// Semantics kept from the reference: beta == 1 adds alpha*op(A)op(B) with
// atomics (C of different entries may alias, kgemm_nt.hpp:184-187),
// beta == 0 stores without reading C, any other beta is a read-modify-write.
//
// Design: entries up to 64 x 64 x 64 run on the FP64 tensor cores
// (kgemm_dmma_kernel, below).  Larger entries: one 64x64 output
// tile per block (16x16 threads, 4x4 outputs per thread), K staged through
// shared memory in steps of 16 with the operand transposes folded into the
// staging loads, FP64 FMA accumulation.
#include <algorithm>
#include <cstdlib>

#include "kron_launch.h"

namespace kron {

namespace {

constexpr int TM = 64, TN = 64, TK = 16;

template <int OP> // 0 = nn, 1 = nt, 2 = tt
__global__ void __launch_bounds__(256)
    kgemm_batched_kernel(int mm, int nn, int kk, double alpha, double *const *Aarr,
                         const int *ldAarr, double *const *Barr, const int *ldBarr, double beta,
                         double *const *Carr, const int *ldCarr, int batch, int tiles_m,
                         int tiles_n)
{
  __shared__ double As[TK][TM + 1];
  __shared__ double Bs[TK][TN + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const long long ntiles = (long long)tiles_m * tiles_n;

  for (long long job = blockIdx.x; job < ntiles * batch; job += gridDim.x)
  {
    const int k    = (int)(job / ntiles);
    const int tile = (int)(job - (long long)k * ntiles);
    const int i0 = (tile % tiles_m) * TM, j0 = (tile / tiles_m) * TN;
    const double *A = Aarr[k];
    const double *B = Barr[k];
    double *C       = Carr[k];
    const long long ldA = ldAarr[k], ldB = ldBarr[k], ldC = ldCarr[k];

    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++)
        acc[a][b] = 0.0;

    for (int k0 = 0; k0 < kk; k0 += TK)
    {
      __syncthreads();
      // op(A) tile: rows i0..i0+63, cols k0..k0+15
      for (int q = threadIdx.x; q < TM * TK; q += 256)
      {
        int i, kq;
        if (OP == 2)
        { // A^T: element (i, kq) = A[kq + i*ldA]; consecutive threads walk kq
          kq = q % TK;
          i  = q / TK;
        }
        else
        { // element (i, kq) = A[i + kq*ldA]; consecutive threads walk i
          i  = q % TM;
          kq = q / TM;
        }
        const int gi = i0 + i, gk = k0 + kq;
        double v     = 0.0;
        if (gi < mm && gk < kk)
          v = (OP == 2) ? A[gk + gi * ldA] : A[gi + gk * ldA];
        As[kq][i] = v;
      }
      // op(B) tile: rows k0..k0+15, cols j0..j0+63
      for (int q = threadIdx.x; q < TK * TN; q += 256)
      {
        int j, kq;
        if (OP == 0)
        { // element (kq, j) = B[kq + j*ldB]
          kq = q % TK;
          j  = q / TK;
        }
        else
        { // B^T: element (kq, j) = B[j + kq*ldB]
          j  = q % TN;
          kq = q / TN;
        }
        const int gj = j0 + j, gk = k0 + kq;
        double v     = 0.0;
        if (gj < nn && gk < kk)
          v = (OP == 0) ? B[gk + gj * ldB] : B[gj + gk * ldB];
        Bs[kq][j] = v;
      }
      __syncthreads();
#pragma unroll
      for (int kq = 0; kq < TK; kq++)
      {
        double a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
        {
          a[u] = As[kq][tx + 16 * u];
          b[u] = Bs[kq][ty + 16 * u];
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
          for (int w = 0; w < 4; w++)
            acc[u][w] = fma(a[u], b[w], acc[u][w]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int w = 0; w < 4; w++)
      {
        const int gi = i0 + tx + 16 * u, gj = j0 + ty + 16 * w;
        if (gi < mm && gj < nn)
        {
          double *c = C + gi + gj * ldC;
          if (beta == 1.0)
            atomicAdd(c, alpha * acc[u][w]);
          else if (beta == 0.0)
            *c = alpha * acc[u][w];
          else
            *c = beta * (*c) + alpha * acc[u][w];
        }
      }
  }
}

// ---------------------------------------------------------------------------
// Entries up to 64 x 64 x 64 on the FP64 tensor cores (mma.sync m16n8k8: half
// the instructions of m8n8k4 at the same rate).  Four warps per entry, or one
// (mm, nn <= 32), so that small entries fill an SM.  A warp holds TM x TN tiles
// of 16 x 8 in fragments, 32 accumulators a lane: 32 x 32 of C, or 16 x 64, or 64 x
// 16, as pick_dmma says.
//
// op(A) and op(B) are staged in shared memory line by line as they lie in
// memory (lines of `len` contiguous elements), at a line stride of 4 mod 16
// elements, so that the fragment reads of either orientation are conflict
// free (a half-warp's 16 lanes hit words 4g + t or 4t + g mod 16).  The
// padding to whole tiles is zeroed once: no copy ever writes there.  The next
// entry's operands (copied 16 bytes at a time where alignment allows) take
// off before the current entry's products when two stages leave enough blocks
// an SM, else before its results go out; its pointers come an entry earlier
// still.
//
// Bound by HBM (64 x 64 x 64, 32768 entries: 4.3 GB, 0.66 ms; FP64 0.46).  Measured
// there 1.20 -> 0.86 ms, 8 x 8 x 8 (60000 entries) 536 -> 52 us, 32 x 32 x 32 (60000)
// 1017 -> 319 us, 58 x 35 x 29 (30000, beta = 0.5) 1382 -> 523 us, against one
// entry a block whatever its size, loads, products and results in series, and two
// divisions per copied element.
constexpr int DM_THREADS = 128;
constexpr int DM_MAX     = 64;

__device__ __forceinline__ void dm_mma(double (&c)[4], const double (&a)[4], const double (&b)[2])
{
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
               "{%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// One operand: `lines` lines of `len` elements, staged at stride S; the magics
// divide by len / 2 and by len (0 for a divisor of 1).
struct DmOperand
{
  int lines, len, S;
  unsigned magic2, magic1;
};

struct DmArgs
{
  int mm, nn, kk, batch;
  DmOperand a, b;
  int a_elems, stage_elems, stages; // shared elements: of op(A), of a stage
  double alpha, beta;
  double *const *A, *const *B, *const *C;
  const int *ldA, *ldB, *ldC;
};

__device__ __forceinline__ void dm_copy(const DmOperand &o, double *dst, const double *src,
                                        long long ld, int t, int G)
{
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0 && (ld & 1) == 0)
  {
    const int units = o.len >> 1;
    for (int q = t; q < o.lines * units; q += G)
    {
      const int l = o.magic2 ? (int)__umulhi((unsigned)q, o.magic2) : q, u = q - l * units;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + l * o.S + 2 * u)),
                   "l"(src + l * ld + 2 * u)
                   : "memory");
    }
    if (o.len & 1)
      for (int l = t; l < o.lines; l += G)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst + l * o.S + o.len - 1)),
                     "l"(src + l * ld + o.len - 1)
                     : "memory");
  }
  else
    for (int q = t; q < o.lines * o.len; q += G)
    {
      const int l = o.magic1 ? (int)__umulhi((unsigned)q, o.magic1) : q, u = q - l * o.len;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst + l * o.S + u)),
                   "l"(src + l * ld + u)
                   : "memory");
    }
}

struct DmEntry
{
  const double *A, *B;
  double *C;
  int ldA, ldB, ldC;
};

__device__ __forceinline__ void dm_entry(const DmArgs &p, int e, DmEntry &d)
{
  d.A   = p.A[e];
  d.B   = p.B[e];
  d.C   = p.C[e];
  d.ldA = p.ldA[e];
  d.ldB = p.ldB[e];
  d.ldC = p.ldC[e];
}

// OP: 0 = nn, 1 = nt, 2 = tt.  WM x WN warps an entry, each with TM x TN tiles;
// FULL: every tile of every warp is whole.
template <int OP, int WM, int WN, int TM, int TN, bool FULL>
__global__ void __launch_bounds__(DM_THREADS, 3)
    kgemm_dmma_kernel(const __grid_constant__ DmArgs p)
{
  extern __shared__ __align__(16) double dm_smem[];
  constexpr int WPE = WM * WN, G = 32 * WPE, NG = DM_THREADS / G;
  const int grp = threadIdx.x / G, tid = threadIdx.x - grp * G;
  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int kt = (p.kk + 7) >> 3;
  const int r0 = (warp / WN) * TM * 16, c0 = (warp % WN) * TN * 8; // this warp's part of C
  // its tiles in use
  const int na = FULL ? TM : min(TM, max(0, (p.mm - r0 + 15) >> 4));
  const int nb = FULL ? TN : min(TN, max(0, (p.nn - c0 + 7) >> 3));
  constexpr bool A_KM = OP != 2; // A staged [k][i], else [i][k]
  constexpr bool B_NK = OP == 0; // B staged [j][k], else [k][j]
  double *base = dm_smem + (size_t)grp * p.stages * p.stage_elems;
  auto sync    = [&]() {
    if constexpr (WPE == 4)
      __syncthreads();
    else
      __syncwarp();
  };

  for (int q = tid; q < p.stages * p.stage_elems; q += G)
    base[q] = 0.0;
  const int step = gridDim.x * NG;
  int e          = blockIdx.x * NG + grp;
  if (e >= p.batch)
    return; // WPE = 1: the warps of a block share no barrier
  sync();
  DmEntry cur, nxt;
  dm_entry(p, e, cur);
  auto issue = [&](const DmEntry &d, int s) {
    double *st = base + s * p.stage_elems;
    dm_copy(p.a, st, d.A, d.ldA, tid, G);
    dm_copy(p.b, st + p.a_elems, d.B, d.ldB, tid, G);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(cur, 0);
  if (e + step < p.batch)
    dm_entry(p, e + step, nxt);
  for (int s = 0;; s ^= p.stages - 1)
  {
    const bool more = e + step < p.batch;
    if (more && p.stages == 2)
    {
      issue(nxt, s ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    }
    else
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    sync();

    // element (row r0 + g, k = t) of op(A), (k = t, column c0 + g) of op(B);
    // steps between rows / columns and between ks
    const int ar = A_KM ? 1 : p.a.S, ak = A_KM ? p.a.S : 1;
    const int bc = B_NK ? p.b.S : 1, bk = B_NK ? 1 : p.b.S;
    const double *Ap = base + s * p.stage_elems + (r0 + g) * ar + t * ak;
    const double *Bp = base + s * p.stage_elems + p.a_elems + (c0 + g) * bc + t * bk;
    double acc[TM][TN][4];
#pragma unroll
    for (int a = 0; a < TM; a++)
#pragma unroll
      for (int b = 0; b < TN; b++)
        acc[a][b][0] = acc[a][b][1] = acc[a][b][2] = acc[a][b][3] = 0.0;
    for (int ks = 0; ks < kt; ks++, Ap += 8 * ak, Bp += 8 * bk)
    {
      double af[TM][4], bf[TN][2];
#pragma unroll
      for (int a = 0; a < TM; a++)
        if (FULL || a < na)
        {
          af[a][0] = Ap[a * 16 * ar];
          af[a][1] = Ap[(a * 16 + 8) * ar];
          af[a][2] = Ap[a * 16 * ar + 4 * ak];
          af[a][3] = Ap[(a * 16 + 8) * ar + 4 * ak];
        }
#pragma unroll
      for (int b = 0; b < TN; b++)
        if (FULL || b < nb)
        {
          bf[b][0] = Bp[b * 8 * bc];
          bf[b][1] = Bp[b * 8 * bc + 4 * bk];
        }
#pragma unroll
      for (int b = 0; b < TN; b++)
        if (FULL || b < nb) // warp-uniform
#pragma unroll
          for (int a = 0; a < TM; a++)
            if (FULL || a < na)
              dm_mma(acc[a][b], af[a], bf[b]);
    }
    sync(); // the stage is read
    double *C           = cur.C + (r0 + g) + (long long)(c0 + 2 * t) * cur.ldC;
    const long long ldc = cur.ldC;
    if (more)
    {
      cur = nxt;
      if (p.stages == 1)
        issue(nxt, 0);
      if (e + 2 * step < p.batch)
        dm_entry(p, e + 2 * step, nxt);
    }
    // acc[a][b][2 h + pp]: row 16 a + 8 h + g, column 8 b + 2 t + pp
    bool row[TM][2];
#pragma unroll
    for (int a = 0; a < TM; a++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        row[a][h] = FULL || r0 + a * 16 + h * 8 + g < p.mm;
    auto each = [&](int b, auto &&f) {
      // the elements of column tile b that lie in C, down the columns
#pragma unroll
      for (int pp = 0; pp < 2; pp++)
#pragma unroll
        for (int a = 0; a < TM; a++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            if (FULL || (row[a][h] && c0 + b * 8 + 2 * t + pp < p.nn))
              f(C + (b * 8 + pp) * ldc + a * 16 + h * 8, a, 2 * h + pp);
    };
    if (p.beta == 1.0)
    {
#pragma unroll
      for (int b = 0; b < TN; b++)
        if (FULL || b < nb)
          each(b, [&](double *c, int a, int i) { atomicAdd(c, p.alpha * acc[a][b][i]); });
    }
    else if (p.beta == 0.0)
    {
#pragma unroll
      for (int b = 0; b < TN; b++)
        if (FULL || b < nb)
          each(b, [&](double *c, int a, int i) { *c = p.alpha * acc[a][b][i]; });
    }
    else
    {
      constexpr int BC = TM >= 4 ? 1 : 4 / TM; // four tiles of C are read at a time
#pragma unroll
      for (int b0 = 0; b0 < TN; b0 += BC)
        if (FULL || b0 < nb)
        {
          double old[BC][TM][4];
#pragma unroll
          for (int b = 0; b < BC; b++)
            each(b0 + b, [&](double *c, int a, int i) { old[b][a][i] = *c; });
#pragma unroll
          for (int b = 0; b < BC; b++)
            each(b0 + b, [&](double *c, int a, int i) {
              *c = p.beta * old[b][a][i] + p.alpha * acc[a][b0 + b][i];
            });
        }
    }
    if (!more)
      break;
    e += step;
  }
}

DmOperand dm_operand(int lines, int len)
{
  auto magic = [](int v) { return v <= 1 ? 0u : (unsigned)(((1ULL << 32) + v - 1) / v); };
  return DmOperand{lines, len, (len + 15) / 16 * 16 + 4, magic(len / 2), magic(len)};
}

template <int OP, int WM, int WN, int TM, int TN, bool FULL>
int launch_dmma(DmArgs p, cudaStream_t stream)
{
  const void *fn =
      reinterpret_cast<const void *>(&kgemm_dmma_kernel<OP, WM, WN, TM, TN, FULL>);
  constexpr int NG = 4 / (WM * WN);
  // lines padded to whole tiles: 16 rows of A, 8 columns of B, 8 along K
  auto up = [](int n, int q) { return (n + q - 1) / q * q; };
  p.a         = OP == 2 ? dm_operand(p.mm, p.kk) : dm_operand(p.kk, p.mm);
  p.b         = OP == 0 ? dm_operand(p.nn, p.kk) : dm_operand(p.kk, p.nn);
  p.a_elems   = up(p.a.lines, OP == 2 ? 16 : 8) * p.a.S;
  p.stage_elems = p.a_elems + up(p.b.lines, 8) * p.b.S;
  // two stages where they leave as many blocks an SM as the registers do
  const size_t stage = (size_t)p.stage_elems * NG * 8;
  p.stages           = 3 * (2 * stage + 1024) <= (size_t)device_info().smem_per_sm ? 2 : 1;
  const size_t smem  = p.stages * stage;
  int per_sm         = 1;
  if (cached_occupancy(fn, DM_THREADS, smem, &per_sm) != KRON_SUCCESS)
    return KRON_ERROR_LAUNCH;
  const long long grid = std::max<long long>(
      1, std::min<long long>((p.batch + NG - 1) / NG, (long long)device_info().sms * per_sm));
  void *args[] = {&p};
  return cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(DM_THREADS), args, smem, stream) ==
                 cudaSuccess
             ? KRON_SUCCESS
             : KRON_ERROR_LAUNCH;
}

template <int OP>
int pick_dmma(const DmArgs &p, cudaStream_t stream)
{
  const int mt = (p.mm + 15) / 16, nt = (p.nn + 7) / 8;
  if (p.mm == 32 && p.nn == 32)
    return launch_dmma<OP, 1, 1, 2, 4, true>(p, stream);
  if (mt <= 2 && nt <= 4)
    return launch_dmma<OP, 1, 1, 2, 4, false>(p, stream);
  if (p.mm == 64 && p.nn == 64)
    return launch_dmma<OP, 2, 2, 2, 4, true>(p, stream);
  // Tiles of the busiest warp: two by two warps of 2 x 4 tiles, four along the
  // rows (1 x 8), four along the columns (4 x 2; rated as if its warps shared
  // the tile columns evenly).  That decides at 3 x 4 tiles only, where two warps
  // of 3 x 2 are faster than three of 1 x 4 (fewer shared-memory loads a product:
  // 16 for 6 against 12 for 4 a K step; 20000 entries, beta = 1 / 0: 48 x 32 x 40
  // 279 / 234 against 315 / 294 us, 40 x 30 x 64 372 / 330 against 401 / 375; only
  // K = 8 is slower, 48 x 28 x 8 162 / 110 against 136 / 110).
  const int t22 = std::min(mt, 2) * std::min(nt, 4), t41 = nt, t14 = mt * ((nt + 3) / 4);
  if (t41 < t22 && t41 <= t14)
    return launch_dmma<OP, 4, 1, 1, 8, false>(p, stream);
  if (t14 < t22)
    return launch_dmma<OP, 1, 4, 4, 2, false>(p, stream);
  return launch_dmma<OP, 2, 2, 2, 4, false>(p, stream);
}

} // namespace

int launch_kgemm(int op, int mm, int nn, int kk, double alpha, double *const *A, const int *ldA,
                 double *const *B, const int *ldB, double beta, double *const *C,
                 const int *ldC, int batch, cudaStream_t stream)
{
  if (batch <= 0 || mm <= 0 || nn <= 0)
    return KRON_SUCCESS;
  // entries up to 64 x 64 x 64 (the reference tests' sizes) on the FP64
  // tensor cores, a block or (up to 32 x 32) a warp an entry
  if (mm <= DM_MAX && nn <= DM_MAX && kk <= DM_MAX && !std::getenv("KRON_KGEMM_CUDA_CORES"))
  {
    DmArgs p{};
    p.mm    = mm;
    p.nn    = nn;
    p.kk    = kk;
    p.batch = batch;
    p.alpha = alpha;
    p.beta  = beta;
    p.A     = A;
    p.B     = B;
    p.C     = C;
    p.ldA   = ldA;
    p.ldB   = ldB;
    p.ldC   = ldC;
    switch (op)
    {
    case 0: return pick_dmma<0>(p, stream);
    case 1: return pick_dmma<1>(p, stream);
    case 2: return pick_dmma<2>(p, stream);
    default: return KRON_ERROR_INVALID_VALUE;
    }
  }
  const int tiles_m = (mm + TM - 1) / TM, tiles_n = (nn + TN - 1) / TN;
  const long long jobs = (long long)tiles_m * tiles_n * batch;
  const int sms        = device_info().sms;
  long long grid       = std::min<long long>(jobs, (long long)sms * 8);
  if (grid < 1)
    grid = 1;
  switch (op)
  {
  case 0:
    kgemm_batched_kernel<0><<<(unsigned)grid, 256, 0, stream>>>(
        mm, nn, kk, alpha, A, ldA, B, ldB, beta, C, ldC, batch, tiles_m, tiles_n);
    break;
  case 1:
    kgemm_batched_kernel<1><<<(unsigned)grid, 256, 0, stream>>>(
        mm, nn, kk, alpha, A, ldA, B, ldB, beta, C, ldC, batch, tiles_m, tiles_n);
    break;
  case 2:
    kgemm_batched_kernel<2><<<(unsigned)grid, 256, 0, stream>>>(
        mm, nn, kk, alpha, A, ldA, B, ldB, beta, C, ldC, batch, tiles_m, tiles_n);
    break;
  default: return KRON_ERROR_INVALID_VALUE;
  }
  return cudaGetLastError() == cudaSuccess ? KRON_SUCCESS : KRON_ERROR_LAUNCH;
}

} // namespace kron
