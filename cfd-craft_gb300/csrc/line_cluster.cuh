// Block Gauss-Seidel sweeps of anisotropic levels on one thread-block cluster (included by
// engine.cu).
//
// A sweep solves its blocks (lines along the stiff axis, or small planes; setup.hpp
// LineBlocks) in the dependency levels of the block order; blocks of one level share no
// entry. A block's banded substitution is a serial chain of 2 len (1 + 2 bw) FP64 operations
// of about 39 ns each, whatever the number of active lanes: 11.2 us for 48 rows of
// half-bandwidth 1, which bounds the sweep (95 levels on a 48 x 48 arrangement of lines). So
// everything else is kept off that chain. Block g of the sweep belongs to thread block g % nb,
// warp (g / nb) % LCW: a level's blocks meet different FP64 pipes, and every warp walks its own
// blocks in order, with their records copied to shared memory one block ahead. The products of
// a block's outside entries are spread over the lanes; those with blocks behind it in the sweep
// are formed, and its right-hand side loaded, before its level begins. The iterate stays in the
// cluster's shared memory (SHX), where the substitution runs in place; levels that do not fit
// there keep it in global memory. One sweep of 48^3 rows: 1.3 ms (13.4 us a level); of the
// 24 x 24 x 2 level with 40 entries a row 0.31 ms (with the entries taken one after the other
// 0.65 ms). The cycle of 48^3 cells, thickness 0.1: 25 -> 10 ms, with the gauges' share cut from
// 4.7 to 0.7 ms of it (engine.cu k_center_sums).
//
// Backward sweeps take the forward dependency levels in reverse: adjacent blocks lie in
// different levels, the lower block in the lower one. Every row sees the operations of the
// sequential loop (multigrid/line.rs:155-190) in its order, so the bits are the reference's.
#pragma once
#include <cooperative_groups.h>

#include "plain_cluster.cuh"
#include "state.hpp"

namespace {

constexpr int LCW = 4;               // warps per block: one per FP64 pipe
constexpr int LCT = 32 * LCW;
constexpr int LC_SMEM = 208 * 1024;  // dynamic shared memory a sweep may ask for

// The banded forward and backward substitutions of one block (multigrid/line.rs:172-185)
// for a half-bandwidth BW: the last BW results stay in registers and the next row's values are
// loaded ahead of the chain. Rows before the first and after the last give products of zeros; PAD:
// the factor has BW rows of zeros behind the last one, else they are left out of the loads.
template <int BW, bool PAD>
__device__ __forceinline__ void line_subst(double* s, const double* fac, int len) {
  constexpr int W = BW + 1;
  struct {
    const double* p;
    int end;
    __device__ __forceinline__ double operator[](int k) const { return PAD || k < end ? p[k] : 0.0; }
  } const f{fac, len * W};
  double w[BW], c[W], n[W];  // w[d]: the result d + 1 rows back (forward) or ahead (backward)
#pragma unroll
  for (int d = 0; d < BW; ++d) w[d] = 0.0;
#pragma unroll
  for (int d = 0; d < W; ++d) c[d] = f[d];
  double v = s[0];
#pragma unroll 4
  for (int i = 0; i < len; ++i) {
    const double vn = s[min(i + 1, len - 1)];
#pragma unroll
    for (int d = 0; d < W; ++d) n[d] = f[(i + 1) * W + d];
#pragma unroll
    for (int d = BW; d >= 1; --d) v = v - c[d] * w[d - 1];  // columns i-BW .. i-1, ascending
    v = v * c[0];
    s[i] = v;
#pragma unroll
    for (int d = BW - 1; d >= 1; --d) w[d] = w[d - 1];
    w[0] = v;
    v = vn;
#pragma unroll
    for (int d = 0; d < W; ++d) c[d] = n[d];
  }
#pragma unroll
  for (int d = 0; d < BW; ++d) w[d] = 0.0;
  v = s[len - 1];
  c[0] = f[(len - 1) * W];
#pragma unroll
  for (int d = 1; d < W; ++d) c[d] = f[(len - 1 + d) * W + d];
#pragma unroll 4
  for (int i = len - 1; i >= 0; --i) {
    const int j = i > 0 ? i - 1 : 0;
    const double vn = s[j];
    n[0] = f[j * W];
#pragma unroll
    for (int d = 1; d < W; ++d) n[d] = f[(j + d) * W + d];
#pragma unroll
    for (int d = 1; d <= BW; ++d) v = v - c[d] * w[d - 1];  // columns i+1 .. i+BW, ascending
    v = v * c[0];
    s[i] = v;
#pragma unroll
    for (int d = BW - 1; d >= 1; --d) w[d] = w[d - 1];
    w[0] = v;
    v = vn;
#pragma unroll
    for (int d = 0; d < W; ++d) c[d] = n[d];
  }
}

// Any half-bandwidth, as line.rs:172-185 writes it.
__device__ __noinline__ void line_subst_any(double* s, const double* f, int len, int bw) {
  const int W = bw + 1;
  for (int i = 0; i < len; ++i) {
    double v = s[i];
    for (int j = max(0, i - bw); j < i; ++j) v = v - f[i * W + i - j] * s[j];
    s[i] = v * f[i * W];
  }
  for (int i = len - 1; i >= 0; --i) {
    double v = s[i];
    for (int j = i + 1; j < min(len, i + bw + 1); ++j) v = v - f[j * W + j - i] * s[j];
    s[i] = v * f[i * W];
  }
}
template <bool PAD>
__device__ __forceinline__ void line_solve(double* s, const double* f, int len, int bw) {
  switch (bw) {
    case 1: line_subst<1, PAD>(s, f, len); break;
    case 2: line_subst<2, PAD>(s, f, len); break;
    case 3: line_subst<3, PAD>(s, f, len); break;
    case 4: line_subst<4, PAD>(s, f, len); break;
    default: line_subst_any(s, f, len, bw); break;
  }
}

// One sweep. Forward sweeps with SHX start from a zero iterate, the others from L.x.
template <bool BWD, bool SHX>
__global__ void __launch_bounds__(LCT, 1) k_line_sweep(LineLev L, const Scalars* S) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (S && S->done) return;  // the whole cluster
  const int rank = (int)cg::this_cluster().block_rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int len = L.len, step = L.nb * LCW;
  int* st = reinterpret_cast<int*>(smem);
  double* xs = reinterpret_cast<double*>(smem + L.x_at);
  unsigned char* buf = smem + L.buf_at + (size_t)warp * 2 * L.rec;
  // The warp's products and (not SHX) the rows it solves.
  double* prod = (L.staged ? reinterpret_cast<double*>(smem + L.scr_at) : L.scr + (size_t)rank * LCW * L.scr_len) +
                 (size_t)warp * L.scr_len;
  double* scr = prod + L.wide * len;
  const unsigned base = pc_addr(smem);
  for (int e = threadIdx.x; e <= L.ndep; e += LCT) st[e] = L.start[e];
  auto rows_of = [&](int g) { return reinterpret_cast<const int*>(L.recs + (size_t)g * L.rec + L.row_at); };
  if (SHX) {
    for (int q = warp; rank + q * L.nb < L.count; q += LCW) {
      const int* rows = rows_of(rank + q * L.nb);
      for (int i = lane; i < len; i += 32) xs[q * len + i] = BWD ? L.x[rows[i]] : 0.0;
    }
    if (threadIdx.x == 0) xs[(L.count + L.nb - 1) / L.nb * len] = 0.0;
  }
  // The warp's blocks, g, g + step, ... (backward: descending); k counts them.
  const int first = rank + L.nb * warp;
  const int dir = BWD ? -step : step;
  int g = BWD ? (L.count > first ? first + (L.count - 1 - first) / step * step : -1) : first, k = 0;
  const auto valid = [&](int h) { return h >= 0 && h < L.count; };
  const auto stage = [&](int h, int which) {  // copies the record of block h ahead
    if (valid(h)) {
      const unsigned char* src = L.recs + (size_t)h * L.rec;
      const unsigned dst = pc_addr(buf + (size_t)which * L.rec);
      for (int o = lane * 16; o < L.rec; o += 512)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + o), "l"(src + o) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const auto record = [&]() { return L.staged ? buf + (size_t)(k & 1) * L.rec : L.recs + (size_t)g * L.rec; };
  // The products of the outside entries [a, b) of the record to their places; lanes behind the
  // last one repeat it.
  const auto products = [&](const unsigned char* rec, int a, int b) {
    const double* val = reinterpret_cast<const double*>(rec + L.val_at);
    const unsigned* col = reinterpret_cast<const unsigned*>(rec + L.col_at);
    const int* place = reinterpret_cast<const int*>(rec + L.place_at);
    for (int t0 = a; t0 < b; t0 += 128) {
      double x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (t0 + 32 * q >= b) break;
        const unsigned c = col[min(t0 + 32 * q + lane, b - 1)];
        x[q] = SHX ? pc_ld<false>(base, c) : __ldcg(&L.x[c]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (t0 + 32 * q >= b) break;
        const int t = min(t0 + 32 * q + lane, b - 1);
        prod[place[t]] = val[t] * x[q];
      }
    }
  };
  // What block g needs and no block before it changes: its right-hand side (the first 64 rows)
  // and the products with the blocks behind it in the sweep.
  double r0 = 0.0, r1 = 0.0;
  const auto prepare = [&]() {
    if (L.staged) {
      stage(g + dir, (k + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
    }
    const unsigned char* rec = record();
    const int* rows = reinterpret_cast<const int*>(rec + L.row_at);
    if (lane < len) r0 = __ldcg(&L.rhs[rows[lane]]);
    if (lane + 32 < len) r1 = __ldcg(&L.rhs[rows[lane + 32]]);
    const int2 cut = *reinterpret_cast<const int2*>(rec);
    if (BWD) products(rec, cut.x, cut.y);
    else products(rec, 0, cut.x);
  };
  if (L.staged) stage(g, 0);
  __syncthreads();
  pc_arrive();
  pc_wait();
  bool ready = valid(g);
  if (ready) prepare();
  __syncwarp();
  for (int d = 0; d < L.ndep; ++d) {
    const int lo = st[BWD ? L.ndep - 1 - d : d], hi = st[BWD ? L.ndep - d : d + 1];
    while (g >= lo && g < hi) {
      if (!ready) prepare();
      ready = false;
      const unsigned char* rec = record();
      const int2 cut = *reinterpret_cast<const int2*>(rec);
      const int ne = reinterpret_cast<const int*>(rec)[2];
      if (BWD) products(rec, 0, cut.x);
      else products(rec, cut.x, cut.y);
      __syncwarp();
      const int* rows = reinterpret_cast<const int*>(rec + L.row_at);
      double* s = SHX ? xs + (g / L.nb) * len : scr;
      for (int i0 = 0; i0 < len; i0 += 64) {
        // Two rows per lane; lanes without one repeat the last row and keep the result.
        const int ia = i0 + lane, ib = ia + 32;
        const int ja = min(ia, len - 1), jb = min(ib, len - 1);
        const bool two = i0 + 32 < len;  // of the whole warp
        double va = i0 == 0 ? r0 : ia < len ? __ldcg(&L.rhs[rows[ja]]) : 0.0;
        double vb = i0 == 0 ? r1 : ib < len ? __ldcg(&L.rhs[rows[jb]]) : 0.0;
#pragma unroll 4
        for (int e = 0; e < ne; ++e) {
          va = va - prod[e * len + ja];
          if (two) vb = vb - prod[e * len + jb];
        }
        if (ia < len) s[ia] = va;
        if (ib < len) s[ib] = vb;
      }
      __syncwarp();
      if (lane == 0) line_solve<true>(s, reinterpret_cast<const double*>(rec + 16), len, L.bw);
      __syncwarp();
      if (!SHX) {
        for (int i = lane; i < len; i += 32) L.x[rows[i]] = s[i];
        __syncwarp();
      }
      g += dir;
      ++k;
    }
    if (!SHX) __threadfence();
    pc_arrive();
    if (!ready && valid(g)) {
      prepare();
      ready = true;
    }
    pc_wait();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (SHX)
    for (int q = warp; rank + q * L.nb < L.count; q += LCW) {
      const int* rows = rows_of(rank + q * L.nb);
      for (int i = lane; i < len; i += 32) L.x[rows[i]] = xs[q * len + i];
    }
}

// One sweep without records, for grids that their context has room for only so, and for levels
// beyond what a record describes: the block smoother's arrays as the host holds them, the iterate
// in global memory, a block's rows summed by the lanes one entry after the other. In the same order,
// so the same bits. The cycle of 48^3 cells, thickness 0.1: 9.3 ms in 112.0 MB with records, 13.7 ms
// in 101.5 MB without; 470 x 460 x 2 and other blocks of a row or two about half as fast.
template <bool BWD>
__global__ void __launch_bounds__(LCT, 1) k_line_sweep_lean(LineLean L, const Scalars* S) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (S && S->done) return;  // the whole cluster
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, len = L.len;
  const int first = (int)cg::this_cluster().block_rank() + L.nb * warp;
  for (int d = 0; d < L.ndep; ++d) {
    const int q = BWD ? L.ndep - 1 - d : d, hi = __ldg(&L.start[q + 1]);
    for (int t = __ldg(&L.start[q]) + first; t < hi; t += L.nb * LCW) {
      const long long at = (long long)__ldg(&L.order[t]) * len;
      double* s = L.scr ? L.scr + at : reinterpret_cast<double*>(smem) + (size_t)warp * len;
      for (int i = lane; i < len; i += 32) {
        double v = __ldcg(&L.rhs[__ldg(&L.nodes[at + i])]);
        const int end = __ldg(&L.off[at + i + 1]);
#pragma unroll 4
        for (int e = __ldg(&L.off[at + i]); e < end; ++e) v = v - __ldg(&L.val[e]) * __ldcg(&L.x[__ldg(&L.col[e])]);
        s[i] = v;
      }
      __syncwarp();
      if (lane == 0) line_solve<false>(s, L.fac + at * (L.bw + 1), len, L.bw);
      __syncwarp();
      for (int i = lane; i < len; i += 32) L.x[__ldg(&L.nodes[at + i])] = s[i];
      __syncwarp();  // the row is reused by the warp's next block
    }
    __threadfence();
    pc_arrive();
    pc_wait();
  }
}

using LineKernel = void (*)(LineLev, const Scalars*);
inline LineKernel line_kernel(bool backward, bool shx) {
  return backward ? shx ? k_line_sweep<true, true> : k_line_sweep<true, false>
                  : shx ? k_line_sweep<false, true> : k_line_sweep<false, false>;
}

}  // namespace
