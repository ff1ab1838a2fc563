// Coarse levels of the plain V-cycle on one thread-block cluster (included by engine.cu).
//
// A lexicographic Gauss-Seidel sweep over a coarse level is a chain of dependency levels
// (about nx + ny + nz of them): rows of one level do not read each other, and a row reads
// only rows of other levels. Each costs a synchronisation, a gather and the row's FP64 chain.
// With rows, orders and iterate in global memory that was 4.2 us a level (128x128x64: 1,288
// levels a cycle, 5.4 ms). Here a cluster of PCS blocks keeps the iterate and the right-hand
// side in shared memory; each block owns a contiguous range of rows, stored by dependency
// level, so a level's rows are one run of consecutive positions, whose entries the threads
// load while the barrier before it is still closing. Products with neighbours that the sweep
// has not reached are formed before the barrier, too; after it come the new neighbours (from
// their owners' shared memory), the row's sums in the reference's order and the division
// through the reciprocal (div_pre). Bounds: about 21 FP64 operations of 64 cycles per level and
// sub-core (0.65 us) plus the barrier and the gather's latency. Measured: 1.45 us a level, a
// V-cycle 10.8 (with the wave.cuh sweeps: 6.6) -> 3.19 ms at 128x128x64, 4.97 -> 1.57 ms at
// 75x61x37.
//
// Levels whose dependency levels hold few rows run in the first block with block barriers;
// larger ones whose residual would keep the cluster's FP64 pipes busy for longer than a launch
// (PC_GRID_ROWS) only sweep here, with grid-wide kernels for their transfers. Backward sweeps
// take the forward dependency levels in reverse: adjacent rows lie in different levels, the
// lower row in the lower one. Every row sees the operations of the sequential loop in its
// order, so the bits are the reference's.
#pragma once
#include "wave.cuh"

namespace {

constexpr int PCS = 16;             // blocks per cluster (non-portable size)
constexpr int PCT = 128;            // threads per block: a warp per sub-core (its FP64 unit takes an operation in 64 cycles)
constexpr int PC_SMEM = 208 * 1024;  // dynamic shared memory a plan may ask for
// Rows above which a level's transfers are grid-wide kernels. A cycle with them against the cluster's
// own: 128x128x64 (131,000 rows) 3.70 / 3.81 ms, 100x84x50 (52,000) 2.43 / 2.47, 110x80x40 without
// buildings (44,000) 42.6 / 42.7; from 30,000 rows down no difference.
constexpr int PC_GRID_ROWS = 40000;
// Mean rows per dependency level up to which one block sweeps alone. None alone, up to 48, 96, 144
// (ms a cycle): 24x20x16 0.48, 0.43, 0.43, 0.43; 40x36x27 0.91, 0.86, 0.86, 0.97; 100x84x50 2.48,
// 2.44, 2.43, 2.57; up to 400 128x128x64 6.2 instead of 3.7. Wide rows would take more: 110x80x40
// without buildings 46.8, 42.6, 42.6, 37.0.
constexpr int PC_SOLO_ROWS = 96;
constexpr int PC_MAXLEV = 12;

constexpr int PCW = 6;
// A row of at most PCW entries, loaded in six 16-byte pieces: values, diagonal and its reciprocal,
// columns (owner << 24 | byte offset in its shared memory). A regular row has its lower
// neighbours in places 0 .. 2 and the upper ones in 3 .. 5, in order; an irregular one (more
// than three either way: rows next to an aggregate found late) all of them from place 0 on.
// Free places hold +0.0 and the column of a +0.0 in the row's own block: their product is +0.0,
// whose difference leaves every number's bits alone.
struct alignas(16) PcRec {
  double val[PCW], d, rd;
  unsigned col[PCW], irregular, pad;
};
static_assert(sizeof(PcRec) == 96, "six 16-byte loads");

struct PcLev {
  int n, chunk, ndep, solo;  // rows, rows per block, dependency levels, all rows in the first block
  int slots;                 // positions of all owners
  int w;                     // entries per row at most
  int x, rhs;                // offsets in the dynamic shared memory (bytes), the same in every block; x[chunk] is +0.0
  int terminal, nblocks;
  const int* ls;             // [block][ndep + 1]: positions where the dependency levels start
  const int* gid;            // [owner][chunk]: the row at a position
  const struct PcRec* rec;   // [owner][chunk], where w <= PCW; else:
  const unsigned* col;       // [w][owner][chunk]: as PcRec::col
  const double* val;         // [w][owner][chunk]
  const double *diag, *rd;   // [owner][chunk]: diagonal and its reciprocal (recip_of)
  const unsigned short* cnt;  // [owner][chunk]: entries
  // Transfers and vectors in row numbering (DevLevel).
  const int *roff, *rcol, *poff, *pcol;
  const double *rval, *pval;
  double *grhs, *gx, *gres;
  const int *ioff, *idx;
  const long long* foff;
  const double* fac;         // terminal factors
};
struct PcPlan {
  int nl;
  PcLev lv[PC_MAXLEV];
};

__device__ __forceinline__ unsigned pc_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// The value at byte offset `col & 0xffffff` of the dynamic shared memory (at `base` in every block)
// of block col >> 24; LOCAL: of this block.
template <bool LOCAL>
__device__ __forceinline__ double pc_ld(unsigned base, unsigned col) {
  unsigned a = base + (col & 0xffffffu);
  double v;
  if (LOCAL) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  } else {
    asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(col >> 24));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  }
  return v;
}
// The aligned forms ask for the whole warp to be at the instruction together, which nothing else
// promises behind a predicated store, the branch of div_rare or a loop of a few lanes.
__device__ __forceinline__ void pc_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void pc_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// v / d through the reciprocal; the extra correction where some lane of the warp needs it.
__device__ __forceinline__ double pc_div(double v, double d, double rd, bool on) {
  return __any_sync(0xffffffffu, on && __double2hiint(rd) < 0) ? div_pre<true>(v, d, rd, on) : div_pre<false>(v, d, rd, on);
}

struct PcRow {
  PcRec r;
  int p;  // position, -1: none
};
__device__ __forceinline__ void pc_fetch(const PcRec* rec, int p, int end, PcRow& R) {
  R.p = p < end ? p : -1;
  if (p >= end) return;
  const uint4* src = reinterpret_cast<const uint4*>(rec + p);
  uint4* dst = reinterpret_cast<uint4*>(&R.r);
#pragma unroll
  for (int m = 0; m < 6; ++m) dst[m] = __ldg(&src[m]);
}

// One sweep of a level by the blocks that own its rows. LOCAL: the first block alone. The rows
// of the next PC_AHEAD dependency levels are in registers or on their way: an L2 round trip
// is about as long as a dependency level.
constexpr int PC_AHEAD = 2;
template <bool BWD, bool LOCAL>
__device__ __noinline__ void pc_sweep_rows(const PcLev& L, int rank, const int* ls, unsigned char* smem) {
  double* x = reinterpret_cast<double*>(smem + L.x);
  const double* rhs = reinterpret_cast<const double*>(smem + L.rhs);
  const PcRec* rec = L.rec + (size_t)rank * L.chunk;
  const unsigned base = pc_addr(smem), zero = (unsigned)rank << 24 | (unsigned)(L.x + 8 * L.chunk);
  const int ndep = L.ndep;
  auto level = [&](int q) { return BWD ? ndep - 1 - q : q; };
  // A row's update, with the barrier before its dependency level between the products with
  // neighbours the sweep has not reached (their values are the previous sweep's) and the
  // others; a warp with an irregular row forms them all after it. A warp without rows stays
  // off the FP64 pipe.
  auto update = [&](PcRow& R, bool barrier) {
    const bool on = R.p >= 0;
    const bool any = __any_sync(0xffffffffu, on), all_after = __any_sync(0xffffffffu, on && R.r.irregular);
    double pr[PCW];
    double v = on ? rhs[R.p] : 0.0;
    auto product = [&](int a) { pr[a] = R.r.val[a] * pc_ld<LOCAL>(base, on ? R.r.col[a] : zero); };
    if (any && !all_after) {
#pragma unroll
      for (int a = 0; a < 3; ++a) product(BWD ? a : a + 3);
      if (BWD) v = v - pr[0] - pr[1] - pr[2];
    }
    if (barrier) {
      if (LOCAL) __syncthreads();
      else pc_wait();
    }
    if (!any) return;
    if (all_after) {
#pragma unroll
      for (int a = 0; a < PCW; ++a) product(a);
      if (BWD) v = v - pr[0] - pr[1] - pr[2];
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a) product(BWD ? a + 3 : a);
    }
    if (!BWD) v = v - pr[0] - pr[1] - pr[2];
    v = v - pr[3] - pr[4] - pr[5];
    // d = 0: an isolated sealed cell, a null pressure space.
    const bool some = on && ((unsigned)__double2hiint(R.r.d) << 1 | (unsigned)__double2loint(R.r.d)) != 0;
    v = pc_div(v, R.r.d, R.r.rd, some);
    if (on) x[R.p] = some ? v : 0.0;
  };
  PcRow R[PC_AHEAD];
  auto fetch = [&](int q, PcRow& S) {
    if (q < ndep) pc_fetch(rec, ls[level(q)] + (int)threadIdx.x, ls[level(q) + 1], S);
  };
#pragma unroll
  for (int m = 0; m < PC_AHEAD; ++m) fetch(m, R[m]);
  for (int q0 = 0; q0 < ndep; q0 += PC_AHEAD) {
#pragma unroll
    for (int m = 0; m < PC_AHEAD; ++m) {
      const int q = q0 + m;
      if (q >= ndep) break;
      update(R[m], q > 0);
      // Further rows of a level with more of them than threads.
      for (int p0 = ls[level(q)] + PCT; p0 < ls[level(q) + 1]; p0 += PCT) {
        PcRow S;
        pc_fetch(rec, p0 + (int)threadIdx.x, ls[level(q) + 1], S);
        update(S, false);
      }
      if (!LOCAL) pc_arrive();
      fetch(q + PC_AHEAD, R[m]);
    }
  }
  if (LOCAL) __syncthreads();
  else pc_wait();
}

// Rows of any width: eight entries' columns and values in flight at a time.
template <bool BWD, bool LOCAL>
__device__ __noinline__ void pc_sweep_wide(const PcLev& L, int rank, const int* ls, unsigned char* smem) {
  double* x = reinterpret_cast<double*>(smem + L.x);
  const double* rhs = reinterpret_cast<const double*>(smem + L.rhs);
  const unsigned base = pc_addr(smem);
  const int stride = L.slots;
  for (int q = 0; q < L.ndep; ++q) {
    const int dep = BWD ? L.ndep - 1 - q : q;
    for (int p0 = ls[dep]; p0 < ls[dep + 1]; p0 += PCT) {
      const int p = p0 + threadIdx.x;
      const bool on = p < ls[dep + 1];
      const int i = rank * L.chunk + p;
      const int cnt = on ? (int)__ldg(&L.cnt[i]) : 0;
      double v = on ? rhs[p] : 0.0;
      for (int a0 = 0; a0 < L.w; a0 += 8) {
        double val[8];
        unsigned col[8];
#pragma unroll
        for (int a = 0; a < 8; ++a)
          if (a0 + a < cnt) {
            val[a] = __ldg(&L.val[(size_t)(a0 + a) * stride + i]);
            col[a] = __ldg(&L.col[(size_t)(a0 + a) * stride + i]);
          }
#pragma unroll
        for (int a = 0; a < 8; ++a)
          if (a0 + a < cnt) v = v - val[a] * pc_ld<LOCAL>(base, col[a]);
      }
      const double d = on ? __ldg(&L.diag[i]) : 0.0, rd = on ? __ldg(&L.rd[i]) : 0.0;
      if (__any_sync(0xffffffffu, on)) v = pc_div(v, d, rd, d != 0.0);
      if (on) x[p] = d != 0.0 ? v : 0.0;
    }
    if (LOCAL) {
      __syncthreads();
    } else {
      pc_arrive();
      pc_wait();
    }
  }
}

template <bool BWD>
__device__ void pc_sweep_level(const PcLev& L, int rank, int* ls, unsigned char* smem) {
  if (L.solo && rank != 0) return;
  __syncthreads();
  for (int e = threadIdx.x; e <= L.ndep; e += PCT) ls[e] = __ldg(&L.ls[rank * (L.ndep + 1) + e]);
  __syncthreads();
  if (L.rec) {
    if (L.solo) pc_sweep_rows<BWD, true>(L, rank, ls, smem);
    else pc_sweep_rows<BWD, false>(L, rank, ls, smem);
  } else {
    if (L.solo) pc_sweep_wide<BWD, true>(L, rank, ls, smem);
    else pc_sweep_wide<BWD, false>(L, rank, ls, smem);
  }
}

// The dense Cholesky solve of a terminal block by one warp (masked.rs:52-69): forward, each
// lane keeps its row and takes the solved ones off in ascending order; backward, the lanes
// form a row's products and every lane runs the row's subtractions in ascending order. Blocks
// of more than 32 rows by one thread.
__device__ __noinline__ void pc_direct(const int* ix, int n, const double* f, const double* rhs, double* x) {
  const int ln = threadIdx.x & 31;
  if (n > 32) {
    if (ln == 0) {
      for (int i = 0; i < n; ++i) {
        double v = rhs[ix[i]];
        for (int j = 0; j < i; ++j) v = v - f[i * n + j] * x[ix[j]];
        x[ix[i]] = v / f[i * n + i];
      }
      for (int i = n - 1; i >= 0; --i) {
        double v = x[ix[i]];
        for (int j = i + 1; j < n; ++j) v = v - f[j * n + i] * x[ix[j]];
        x[ix[i]] = v / f[i * n + i];
      }
    }
    return;
  }
  const bool on = ln < n;
  const double d = on ? __ldg(&f[ln * n + ln]) : 1.0, rd = recip_of(d);
  double v = on ? rhs[ix[ln]] : 0.0, s = 0.0;
  double fj = on && ln > 0 ? __ldg(&f[ln * n]) : 0.0;
  for (int j = 0; j < n; ++j) {
    const double fn = on && j + 1 < ln ? __ldg(&f[ln * n + j + 1]) : 0.0;  // the next column's entry
    const double xj = __shfl_sync(0xffffffffu, pc_div(v, d, rd, ln == j), j);
    if (ln == j) s = xj;
    if (on && ln > j) v = v - fj * xj;
    fj = fn;
  }
  // s: the forward solution of row ln; x: the backward one.
  double xl = 0.0;
  for (int i = n - 1; i >= 0; --i) {
    const double pr = (on && ln > i ? __ldg(&f[ln * n + i]) : 0.0) * xl;
    double t = __shfl_sync(0xffffffffu, s, i);
    for (int j = i + 1; j < n; ++j) t = t - __shfl_sync(0xffffffffu, pr, j);
    const double di = __shfl_sync(0xffffffffu, d, i), ri = __shfl_sync(0xffffffffu, rd, i);
    t = pc_div(t, di, ri, true);
    if (ln == i) xl = t;
  }
  if (on) x[ix[ln]] = xl;
}

// res = rhs - A x of a level whose transfers are grid-wide, from the plan's rows: the vectors in
// row numbering, the neighbours through their owners' positions.
__global__ void k_plan_residual(const PcPlan* plan, int l, const Scalars* S) {
  if (S && S->done) return;
  const PcLev& L = plan->lv[l];
  const int slots = L.slots;
  const auto at = [&](unsigned c) {  // the value that a place's column names
    const int pos = ((int)(c & 0xffffffu) - L.x) >> 3;
    return pos < L.chunk ? L.gx[__ldg(&L.gid[(int)(c >> 24) * L.chunk + pos])] : 0.0;
  };
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < slots; q += gridDim.x * blockDim.x) {
    if (q % L.chunk >= L.n - q / L.chunk * L.chunk) continue;  // behind the last block's rows
    const int i = __ldg(&L.gid[q]);
    double v;
    if (L.rec) {
      PcRow R;
      pc_fetch(L.rec, q, slots, R);
      v = R.r.d * L.gx[i];
#pragma unroll
      for (int a = 0; a < PCW; ++a) {
        const double t = R.r.val[a] * at(R.r.col[a]);
        v = v + (R.r.val[a] == 0.0 ? -0.0 : t);  // a free place adds -0.0, as below
      }
    } else {
      v = __ldg(&L.diag[q]) * L.gx[i];
      const int cnt = __ldg(&L.cnt[q]);
      for (int a = 0; a < cnt; ++a) v = v + __ldg(&L.val[(size_t)a * slots + q]) * at(__ldg(&L.col[(size_t)a * slots + q]));
    }
    L.gres[i] = L.grhs[i] - v;
  }
}

// what 0: two forward sweeps of level `from` from zero, its iterate to global memory. 1: two
// backward sweeps of its iterate in global memory. 2: the whole cycle from level `from` on.
__global__ void __launch_bounds__(PCT, 1) k_plain_cluster(const PcPlan* plan, int from, int what, const Scalars* S) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PcLev sL, sN;
  if (S && S->done) return;  // the whole cluster
  const int rank = (int)cg::this_cluster().block_rank(), nl = plan->nl;
  int* ls = reinterpret_cast<int*>(smem);  // the dependency level starts of the level being swept
  auto load = [&](int l) {  // the descriptors of level l and the one below
    __syncthreads();
    const int words = (int)(sizeof(PcLev) / 8);
    for (int e = threadIdx.x; e < words; e += PCT) {
      reinterpret_cast<long long*>(&sL)[e] = reinterpret_cast<const long long*>(&plan->lv[l])[e];
      if (l + 1 < nl) reinterpret_cast<long long*>(&sN)[e] = reinterpret_cast<const long long*>(&plan->lv[l + 1])[e];
    }
    __syncthreads();
  };
  auto rows_of = [&](const PcLev& L) { return L.solo ? (rank == 0 ? L.n : 0) : max(0, min(L.chunk, L.n - rank * L.chunk)); };
  int last = what == 2 ? nl - 1 : from;
  if (what != 1) {
    for (int l = from; l <= last; ++l) {
      load(l);
      const PcLev& L = sL;
      double *x = reinterpret_cast<double*>(smem + L.x), *rhs = reinterpret_cast<double*>(smem + L.rhs);
      const int m = rows_of(L);
      for (int p = threadIdx.x; p < m; p += PCT) {
        const int i = L.terminal ? p : __ldg(&L.gid[rank * L.chunk + p]);
        rhs[p] = __ldcg(&L.grhs[i]);
        x[p] = 0.0;
      }
      if (threadIdx.x == 0) x[L.chunk] = 0.0;
      if (L.solo) __syncthreads();
      else cg::this_cluster().sync();
      if (L.terminal) {
        if (rank == 0) {
          for (int bk = threadIdx.x >> 5; bk < L.nblocks; bk += PCT / 32)
            pc_direct(L.idx + L.ioff[bk], L.ioff[bk + 1] - L.ioff[bk], L.fac + L.foff[bk], rhs, x);
          __syncthreads();
          for (int i = threadIdx.x; i < L.n; i += PCT) L.gx[i] = x[i];
        }
        break;
      }
      pc_sweep_level<false>(L, rank, ls, smem);
      pc_sweep_level<false>(L, rank, ls, smem);
      if (what == 0) {
        for (int p = threadIdx.x; p < m; p += PCT) L.gx[__ldg(&L.gid[rank * L.chunk + p])] = x[p];
        return;
      }
      // res = rhs - A x (the row's entries in order), then the restriction.
      const unsigned base = pc_addr(smem);
      const int stride = L.slots;
      for (int p = threadIdx.x; p < m; p += PCT) {
        const int i = rank * L.chunk + p;
        double v;
        if (L.rec) {
          PcRow R;
          pc_fetch(L.rec + (size_t)rank * L.chunk, p, m, R);
          v = R.r.d * x[p];
#pragma unroll
          for (int a = 0; a < PCW; ++a) {
            // A free place adds -0.0 here, which leaves every number alone.
            const double t = R.r.val[a] * pc_ld<false>(base, R.r.col[a]);
            v = v + (R.r.val[a] == 0.0 ? -0.0 : t);
          }
        } else {
          const int cnt = (int)__ldg(&L.cnt[i]);
          v = __ldg(&L.diag[i]) * x[p];
          for (int a0 = 0; a0 < cnt; a0 += 8) {
            double val[8];
            unsigned col[8];
#pragma unroll
            for (int a = 0; a < 8; ++a)
              if (a0 + a < cnt) {
                val[a] = __ldg(&L.val[(size_t)(a0 + a) * stride + i]);
                col[a] = __ldg(&L.col[(size_t)(a0 + a) * stride + i]);
              }
#pragma unroll
            for (int a = 0; a < 8; ++a)
              if (a0 + a < cnt) v = v + val[a] * pc_ld<false>(base, col[a]);
          }
        }
        L.gres[__ldg(&L.gid[i])] = rhs[p] - v;
      }
      __threadfence();
      cg::this_cluster().sync();
      const PcLev& N = sN;
      for (int j = rank * PCT + threadIdx.x; j < N.n; j += PCS * PCT) {
        double v = 0.0;
        for (int k = __ldg(&L.roff[j]); k < __ldg(&L.roff[j + 1]); ++k)
          v = v + __ldg(&L.rval[k]) * __ldcg(&L.gres[__ldg(&L.rcol[k])]);
        N.grhs[j] = v;
      }
      __threadfence();
      cg::this_cluster().sync();
    }
    if (what == 0) return;
    __threadfence();
    cg::this_cluster().sync();
  }
  for (int l = what == 1 ? from : last - 1; l >= from; --l) {
    load(l);
    const PcLev& L = sL;
    double *x = reinterpret_cast<double*>(smem + L.x), *rhs = reinterpret_cast<double*>(smem + L.rhs);
    const int m = rows_of(L);
    for (int p = threadIdx.x; p < m; p += PCT) {
      const int i = __ldg(&L.gid[rank * L.chunk + p]);
      if (what == 1) {
        x[p] = __ldcg(&L.gx[i]);
        rhs[p] = __ldcg(&L.grhs[i]);
      } else {  // x += P x_c
        double s = -0.0;
        for (int k = __ldg(&L.poff[i]); k < __ldg(&L.poff[i + 1]); ++k)
          s = s + __ldg(&L.pval[k]) * __ldcg(&sN.gx[__ldg(&L.pcol[k])]);
        x[p] = x[p] + s;
      }
    }
    if (threadIdx.x == 0) x[L.chunk] = 0.0;
    if (L.solo) __syncthreads();
    else cg::this_cluster().sync();
    pc_sweep_level<true>(L, rank, ls, smem);
    pc_sweep_level<true>(L, rank, ls, smem);
    for (int p = threadIdx.x; p < m; p += PCT) L.gx[__ldg(&L.gid[rank * L.chunk + p])] = x[p];
    __threadfence();
    cg::this_cluster().sync();
  }
}

}  // namespace
