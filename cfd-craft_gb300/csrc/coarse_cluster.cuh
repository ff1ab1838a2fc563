// The coarse levels of one case on one thread-block cluster (included by mixed.cu).
//
// A V-cycle's coarse levels are a chain of some forty short phases (sweep colours, residual
// with restriction, prolongation). Spread over the whole grid each phase costs a grid
// barrier (1.18 us) and two or three dependent round trips to L2; with one cluster of
// CLS blocks per case the barrier is the cluster's (0.3 us) and the iterates stay in the
// blocks' shared memory. Measured per cycle: 128x128x64 (131,072 rows on the first coarse
// level) 256 -> 55 us, 100x84x50 235 -> 45 us, sixteen cases of 128x128x64 368 -> 158 us
// (seven clusters fit the device at once), 8.4 M cells (first level grid-wide) 331 -> 136 us.
// What bounds it now is the chain of barriers and shared-memory round trips.
//
// Levels laid out as the grid of 2x2x2 bins (build_case) are split into slabs of bin layers
// along z, one per block: the last distributed level's layers evenly, the finer levels'
// slabs nested in them (a level's layers 2K, 2K+1 in the block that holds layer K of the
// next), so restriction and prolongation stay inside a block. A block keeps its slab's
// iterate with one halo layer on either side; who updates a boundary layer stores it in the
// neighbour's halo as well (distributed shared memory). A level's rows come in few types (the
// values and positions of a row's entries, its diagonal: 261 among the 131,072 rows of a
// site with 30 buildings), so a row is a 16-bit index into a table in shared memory: three
// 16-byte loads give its six values, six offsets and diagonal. The first distributed level,
// which is the largest, keeps its row types and right-hand side in registers (CLR rows per
// thread and colour), the others in shared memory. From the first level without a bin layout
// on (two aggregates in one bin), the levels of some size are split by rows, with index lists
// and the iterate in global memory (one L2 round trip a phase). Small bin levels and the
// levels below (any aggregation level of at most two colours without closed groups, the
// terminal blocks) run in the cluster's first block with block barriers. Levels too large for
// this run grid-wide: bin levels over their row types (k_up_*), others in the phases of
// k_coarse_all, which hand over at the first cluster level. (Handing over one level later than
// the shared memory asks for was slower: 100x84x50 43 -> 55 us, eight uneven cases 6.73 -> 7.24
// ms a projection.)
//
// Every row sees the operations of the grid-wide phases in the same order (its entries and
// children in the order of the hierarchy), so the results are the same bits (tested against
// the index-list layout).

constexpr int CLS = 16;    // blocks per cluster (non-portable size)
constexpr int CLT = 512;   // threads per block
constexpr int CLR = 16;    // rows per thread and colour of the first distributed level
constexpr int CLB = 6;     // bin levels at most
constexpr int CL_SMEM = 224 * 1024;  // dynamic shared memory a case may ask for

// One bin level. Rows of colour c: bin (I, J, K) with I = 2 s + par, par the parity that makes
// I + J + K + c even, in slot (K nby + J) nbh + s. All offsets are into the dynamic shared
// memory, in bytes, the same in every block of the cluster.
struct ClBin {
  int nby, nbz, nbh, plane, h;  // bins in y and z, slots per bin row, per layer, per colour
  unsigned mh, my;              // bin_magic of nbh and nby
  int layers;                   // layers per block at most
  int x;                        // iterate, [colour][(layers + 2) * plane]
  int rhs, type;                // right-hand side and row types, [colour][layers * plane]; -1: in registers
  int tab, ntypes;              // the row types' table
  const unsigned short* gtype;  // [2h]
  const float4* gtab;           // [ntypes][3], see cl_sum
  const float* grhs;            // the level's right-hand side and iterate in global memory
  float *gx, *gres;
};
struct ClCase {
  int on;            // the case runs here
  int lc, nb, nd;    // first level (index into CCase::lv), bin levels, distributed ones among them
  int ng, ndl;       // further levels after the bins, and how many of them are split by rows (only when nb == nd)
  int slab[CLS + 1]; // layers of the last distributed level per block
  int gx[MAXL], grhs[MAXL];  // the further levels' iterates and right-hand sides (offsets)
  float alpha;       // scale of the coarse corrections
  int smem;          // bytes
  ClBin b[CLB];
};
// The bin levels above the cluster's first one (lv[n], whose right-hand side they give and whose
// iterate they take): grid-wide kernels over the same row types (k_up_*).
constexpr int CLUP = 4;
struct ClUp {
  int n;
  float alpha;
  float* rhs[CLUP + 1];
  ClBin lv[CLUP + 1];
};
static_assert(sizeof(ClCase) % 8 == 0, "ClCase is copied to shared memory in 8-byte words");

// A block's view of a bin level.
struct ClView {
  const ClBin* B;
  int k0, L, nl;        // first layer, layers and rows per colour of this block's slab
  int prev, next;       // blocks holding the layers below and above (-1: none)
  int prevL;            // layers of the block below
  int ldx;              // floats between the colours' iterates
  float* x;             // own iterate of colour 0 (its lower halo layer first)
  float *px, *nx;       // the neighbours' (distributed shared memory)
};

__device__ __forceinline__ void cl_layers(const ClCase& C, int l, int rank, int& k0, int& k1) {
  const ClBin& B = C.b[l];
  if (l >= C.nd) {  // a level of the first block alone
    k0 = 0;
    k1 = rank == 0 ? B.nbz : 0;
    return;
  }
  const int s = C.nd - 1 - l;
  k0 = min(C.slab[rank] << s, B.nbz);
  k1 = min(C.slab[rank + 1] << s, B.nbz);
}

__device__ __forceinline__ ClView cl_view(const ClCase& C, int l, int rank, unsigned char* smem) {
  ClView V;
  V.B = &C.b[l];
  int k1;
  cl_layers(C, l, rank, V.k0, k1);
  V.L = k1 - V.k0;
  V.nl = V.L * V.B->plane;
  V.ldx = (V.B->layers + 2) * V.B->plane;
  V.x = reinterpret_cast<float*>(smem + V.B->x);
  V.prev = V.next = -1;
  V.prevL = 0;
  V.px = V.nx = nullptr;
  if (l < C.nd && V.L > 0) {
    for (int r = rank - 1; r >= 0 && V.prev < 0; --r)
      if (C.slab[r + 1] > C.slab[r]) V.prev = r;
    for (int r = rank + 1; r < CLS && V.next < 0; ++r)
      if (C.slab[r + 1] > C.slab[r]) V.next = r;
    cg::cluster_group cl = cg::this_cluster();
    if (V.prev >= 0) {
      int a, b;
      cl_layers(C, l, V.prev, a, b);
      V.prevL = b - a;
      V.px = cl.map_shared_rank(V.x, V.prev);
    }
    if (V.next >= 0) V.nx = cl.map_shared_rank(V.x, V.next);
  }
  return V;
}

// Stores row q (of the slab) of colour c, and in the neighbours' halos on a boundary layer.
__device__ __forceinline__ void cl_store(const ClView& V, int c, int q, float v) {
  const int P = V.B->plane;
  V.x[c * V.ldx + P + q] = v;
  if (V.px && q < P) V.px[c * V.ldx + (V.prevL + 1) * P + q] = v;
  if (V.nx && q >= V.nl - P) V.nx[c * V.ldx + q - (V.nl - P)] = v;
}

// A row type: entries 0..5 in row order and the offsets of their columns from the row's slot in
// the other colour, diag, 1/diag, the order of the children: {w0, w1, w2, w3}, {w4, w5, diag,
// 1/diag}, {offsets 0 and 1, 2 and 3, 4 and 5 as 16-bit pairs, child order}. Absent entries
// are 0 at offset 0 (some finite value of the slab or its halo).
struct ClRow {
  float4 a, b;
  int4 o;
};
__device__ __forceinline__ ClRow cl_row(const float4* tab, unsigned type) {
  ClRow r;
  r.a = tab[3 * type];
  r.b = tab[3 * type + 1];
  r.o = *reinterpret_cast<const int4*>(&tab[3 * type + 2]);
  return r;
}
__device__ __forceinline__ int cl_off0(int p) { return (int)(short)p; }
__device__ __forceinline__ int cl_off1(int p) { return p >> 16; }
// v + sum over the row's entries of sign w x in row order. xo: the other colour's iterate at
// this row's slot.
template <bool NEG>
__device__ __forceinline__ float cl_sum(float v, const float* xo, const ClRow& r) {
  const float x0 = xo[cl_off0(r.o.x)], x1 = xo[cl_off1(r.o.x)], x2 = xo[cl_off0(r.o.y)], x3 = xo[cl_off1(r.o.y)],
              x4 = xo[cl_off0(r.o.z)], x5 = xo[cl_off1(r.o.z)];
  v = fmaf(NEG ? -r.a.x : r.a.x, x0, v);
  v = fmaf(NEG ? -r.a.y : r.a.y, x1, v);
  v = fmaf(NEG ? -r.a.z : r.a.z, x2, v);
  v = fmaf(NEG ? -r.a.w : r.a.w, x3, v);
  v = fmaf(NEG ? -r.b.x : r.b.x, x4, v);
  v = fmaf(NEG ? -r.b.y : r.b.y, x5, v);
  return v;
}

// ------------------------------------------------------------ the register level
struct ClRegs {
  unsigned type[2][CLR / 2];  // two rows' types each
  float rhs[2][CLR];
  float keep[CLR];  // colour 0's iterate while the residual takes its place
};

template <int C, bool SKIPX>
__device__ __forceinline__ void cl_sweep_reg(const ClView& V, const ClRegs& R, const float4* tab) {
  const int P = V.B->plane;
  const float* __restrict__ xo = V.x + (1 - C) * V.ldx + P;
#pragma unroll
  for (int m = 0; m < CLR; ++m) {
    const int q = threadIdx.x + m * CLT;
    if (q >= V.nl) break;
    const unsigned type = (R.type[C][m / 2] >> (16 * (m & 1))) & 0xffffu;
    float v = R.rhs[C][m], id;
    if (SKIPX) {
      id = tab[3 * type + 1].w;
    } else {
      const ClRow r = cl_row(tab, type);
      v = cl_sum<true>(v, xo + q, r);
      id = r.b.w;
    }
    cl_store(V, C, q, v * id);
  }
}

// Colour 0's residual in place of its iterate, which goes to registers.
__device__ __forceinline__ void cl_resid_reg(const ClView& V, ClRegs& R, const float4* tab) {
  const int P = V.B->plane;
  const float* __restrict__ xo = V.x + V.ldx + P;
#pragma unroll
  for (int m = 0; m < CLR; ++m) {
    const int q = threadIdx.x + m * CLT;
    if (q >= V.nl) break;
    const ClRow r = cl_row(tab, (R.type[0][m / 2] >> (16 * (m & 1))) & 0xffffu);
    const float x = V.x[P + q];
    const float v = cl_sum<false>(__fmul_rn(r.b.z, x), xo + q, r);
    R.keep[m] = x;
    V.x[P + q] = R.rhs[0][m] - v;
  }
}

// ------------------------------------------------------------ levels in shared memory
__device__ __forceinline__ void cl_sweep_smem(const ClView& V, int c, bool skipx, unsigned char* smem) {
  const ClBin& B = *V.B;
  const int rows = B.layers * B.plane, P = B.plane;
  const float* __restrict__ rhs = reinterpret_cast<const float*>(smem + B.rhs) + c * rows;
  const unsigned short* __restrict__ ty = reinterpret_cast<const unsigned short*>(smem + B.type) + c * rows;
  const float4* __restrict__ tab = reinterpret_cast<const float4*>(smem + B.tab);
  const float* __restrict__ xo = V.x + (1 - c) * V.ldx + P;
#pragma unroll 2
  for (int q = threadIdx.x; q < V.nl; q += CLT) {
    const ClRow r = cl_row(tab, ty[q]);
    float v = rhs[q];
    if (!skipx) v = cl_sum<true>(v, xo + q, r);
    cl_store(V, c, q, v * r.b.w);
  }
}
// The residual of row q, colour 0.
__device__ __forceinline__ float cl_resid_smem(const ClView& V, int q, const unsigned char* smem) {
  const ClBin& B = *V.B;
  const int P = B.plane;
  const unsigned short* ty = reinterpret_cast<const unsigned short*>(smem + B.type);
  const ClRow r = cl_row(reinterpret_cast<const float4*>(smem + B.tab), ty[q]);
  const float v = cl_sum<false>(__fmul_rn(r.b.z, V.x[P + q]), V.x + V.ldx + P + q, r);
  return reinterpret_cast<const float*>(smem + B.rhs)[q] - v;
}

// The right-hand side of bin (row q of colour c of the coarse view W) from the colour-0
// residuals of its children, res(k, j, slot); the children of bin (I, J, K) are bins of layers
// 2K, 2K+1 and rows 2J, 2J+1, one of colour 0 in each, all in slot I. order: two bits per
// child in the order of the sum, 2 (k & 1) + (j & 1).
template <class Res>
__device__ __forceinline__ float cl_restrict(const ClView& W, int c, int q, int order, int fine_y, int fine_z, int fine_h,
                                             Res res) {
  const int R = bin_div(q, W.B->mh, W.B->nbh), kk = bin_div(R, W.B->my, W.B->nby);
  const int J = R - kk * W.B->nby, K = W.k0 + kk, s = q - R * W.B->nbh;
  const int I = 2 * s + ((c + J + K) & 1);
  float acc = 0.0f;
  if (I < fine_h) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int ch = order >> (2 * a), k = 2 * K + ((ch >> 1) & 1), j = 2 * J + (ch & 1);
      if (k < fine_z && j < fine_y) acc = acc + res(k, j, I);
    }
  }
  return acc;
}

// The iterate of the parent of colour-0 row q of V in the coarse view W (same block).
__device__ __forceinline__ float cl_parent(const ClView& V, const ClView& W, int q) {
  const int R = bin_div(q, V.B->mh, V.B->nbh), kk = bin_div(R, V.B->my, V.B->nby);
  const int J = R - kk * V.B->nby, K = V.k0 + kk, s = q - R * V.B->nbh;
  const int J1 = J >> 1, K1 = K >> 1, c1 = (s + J1 + K1) & 1;
  return W.x[c1 * W.ldx + W.B->plane + (K1 - W.k0) * W.B->plane + J1 * W.B->nbh + (s >> 1)];
}
// The same through the coarse level's iterate in global memory.
__device__ __forceinline__ float cl_parent_global(const ClView& V, const ClBin& W, int q) {
  const int R = bin_div(q, V.B->mh, V.B->nbh), kk = bin_div(R, V.B->my, V.B->nby);
  const int J = R - kk * V.B->nby, K = V.k0 + kk, s = q - R * V.B->nbh;
  const int J1 = J >> 1, K1 = K >> 1, c1 = (s + J1 + K1) & 1;
  return __ldcg(&W.gx[c1 * W.h + (K1 * W.nby + J1) * W.nbh + (s >> 1)]);
}

// ------------------------------------------------------------ further levels
// Any aggregation level of at most two colours without closed groups, through index lists in
// global memory; the arithmetic of gs_rows/res0_rows. A row's columns and values are loaded
// together (eight in flight), then its neighbours. GLOBAL: the iterate is in global memory.
template <bool GLOBAL, bool NEG>
__device__ __forceinline__ float cl_list_sum(float v, const int* ec, const float* ev, int nrow, int w, const float* x) {
  for (int a0 = 0; a0 < w; a0 += 8) {
    int col[8];
    float val[8], xv[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const bool ok = a0 + a < w;
      col[a] = ok ? __ldg(&ec[(a0 + a) * nrow]) : 0;
      val[a] = ok ? __ldg(&ev[(a0 + a) * nrow]) : 0.0f;
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) xv[a] = GLOBAL ? __ldcg(&x[col[a]]) : x[col[a]];
#pragma unroll
    for (int a = 0; a < 8; ++a)
      if (a0 + a < w) v = fmaf(NEG ? -val[a] : val[a], xv[a], v);
  }
  return v;
}
// One colour's rows t0, t0 + step, ...
template <bool GLOBAL>
__device__ __forceinline__ void cl_sweep_list(const CLev& L, int color, bool skipx, float* x, const float* rhs, int t0,
                                              int step) {
  const int c0 = L.coff[color], nrow = L.coff[color + 1] - c0, base = L.ell_off[color], w = L.ell_w[color];
  for (int t = t0; t < nrow; t += step) {
    float v = GLOBAL ? __ldcg(&rhs[c0 + t]) : rhs[c0 + t];
    const float id = __ldg(&L.idiag[c0 + t]);
    if (!skipx) v = cl_list_sum<GLOBAL, true>(v, L.ell_col + base + t, L.ell_val + base + t, nrow, w, x);
    x[c0 + t] = v * id;
  }
}
template <bool GLOBAL>
__device__ __forceinline__ float cl_resid_list(const CLev& L, int i, const float* x, const float* rhs) {
  const int nrow = L.coff[1], base = L.ell_off[0], w = L.ell_w[0];  // colour 0
  const float xi = GLOBAL ? __ldcg(&x[i]) : x[i];
  const float v = cl_list_sum<GLOBAL, false>(__fmul_rn(__ldg(&L.diag[i]), xi), L.ell_col + base + i, L.ell_val + base + i,
                                             nrow, w, x);
  return (GLOBAL ? __ldcg(&rhs[i]) : rhs[i]) - v;
}
// x_idx = (L L^T)^-1 rhs_idx in FP64, one warp per block (terminal_block).
__device__ __forceinline__ void cl_terminal(const CLev& L, float* x, const float* rhs) {
  const int ln = threadIdx.x & 31;
  for (int bk = threadIdx.x >> 5; bk < L.nblocks; bk += CLT / 32) {
    const int* ix = L.idx + L.ioff[bk];
    const int n = L.ioff[bk + 1] - L.ioff[bk];
    const double* m = L.fac + L.foff[bk];
    const double rj = ln < n ? (double)rhs[ix[ln]] : 0.0;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    for (int j = 0; j < n; j += 4) {
      const double r0 = __shfl_sync(0xffffffffu, rj, j);
      const double r1 = __shfl_sync(0xffffffffu, rj, j + 1 < 32 ? j + 1 : 31);
      const double r2 = __shfl_sync(0xffffffffu, rj, j + 2 < 32 ? j + 2 : 31);
      const double r3 = __shfl_sync(0xffffffffu, rj, j + 3 < 32 ? j + 3 : 31);
      if (ln < n) {
        a0 = fma(m[ln * n + j], r0, a0);
        if (j + 1 < n) a1 = fma(m[ln * n + j + 1], r1, a1);
        if (j + 2 < n) a2 = fma(m[ln * n + j + 2], r2, a2);
        if (j + 3 < n) a3 = fma(m[ln * n + j + 3], r3, a3);
      }
    }
    if (ln < n) x[ix[ln]] = (float)((a0 + a1) + (a2 + a3));
  }
}

// Levels of the first block alone, from the first one that is not split down to the terminal
// level and back: bin levels, then further ones. The right-hand side of the first of them
// comes from the colour-0 residuals of the last split level (or, without one, is the level's
// own in global memory); its iterate goes back to global memory.
__device__ void cl_first_block(const ClCase& C, const CCase& D, int nu, unsigned char* smem) {
  const int nd = C.nd + C.ndl, nb = C.nb, last = nb + C.ng - 1;  // first level, bin levels, the terminal level
  auto lev = [&](int l) -> const CLev& { return D.lv[C.lc + l]; };
  auto lx = [&](int l) { return reinterpret_cast<float*>(smem + C.gx[l]); };
  auto lr = [&](int l) { return reinterpret_cast<float*>(smem + C.grhs[l]); };
  for (int l = nd; l <= last; ++l) {
    const CLev& L = lev(l);
    if (l < nb) {
      const ClView V = cl_view(C, l, 0, smem);
      const ClBin& B = *V.B;
      float* rhs = reinterpret_cast<float*>(smem + B.rhs);
      const int rows = B.layers * B.plane;
      const ClView F = l > nd ? cl_view(C, l - 1, 0, smem) : V;
      auto order = [&](int r) {
        const float4* tab = reinterpret_cast<const float4*>(smem + B.tab);
        return __float_as_int(tab[3 * reinterpret_cast<const unsigned short*>(smem + B.type)[r] + 2].w);
      };
      for (int e = threadIdx.x; e < 2 * V.nl; e += CLT) {
        const int c = e >= V.nl ? 1 : 0, q = e - c * V.nl;
        float v;
        if (l == 0) {
          v = __ldcg(&B.grhs[c * B.h + q]);
        } else if (l == nd) {
          const ClBin& G = C.b[l - 1];
          v = cl_restrict(V, c, q, order(c * rows + q), G.nby, G.nbz, G.nbh,
                          [&](int k, int j, int s) { return __ldcg(&G.gres[(k * G.nby + j) * G.nbh + s]); });
        } else {
          v = cl_restrict(V, c, q, order(c * rows + q), F.B->nby, F.B->nbz, F.B->nbh, [&](int k, int j, int s) {
            return cl_resid_smem(F, (k * F.B->nby + j) * F.B->nbh + s, smem);
          });
        }
        rhs[c * rows + q] = v;
      }
      __syncthreads();
      for (int sw = 0; sw < nu; ++sw)
        for (int c = 0; c < 2; ++c) {
          cl_sweep_smem(V, c, sw == 0 && c == 0, smem);
          __syncthreads();
        }
      continue;
    }
    float *x = lx(l), *rhs = lr(l);
    ClView F;
    if (l > nd && l - 1 < nb) F = cl_view(C, l - 1, 0, smem);
    for (int i = threadIdx.x; i < L.n; i += CLT) {
      float v;
      if (l == 0) {
        v = __ldcg(&L.rhs[i]);
      } else {
        const CLev& M = lev(l - 1);  // its colour-0 children of row i, in order, with weight 1
        v = 0.0f;
        for (int k = M.roff[i]; k < M.roff[i + 1]; ++k) {
          const int ch = M.rchild[k];
          v = v + (l == nd        ? (l - 1 >= nb ? cl_resid_list<true>(M, ch, M.x, M.rhs) : __ldcg(&M.res[ch]))
                   : l - 1 >= nb ? cl_resid_list<false>(M, ch, lx(l - 1), lr(l - 1))
                                 : cl_resid_smem(F, ch, smem));
        }
      }
      rhs[i] = v;
      x[i] = 0.0f;
    }
    __syncthreads();
    if (l == last) {
      cl_terminal(L, x, rhs);
      __syncthreads();
      break;
    }
    for (int sw = 0; sw < nu; ++sw)
      for (int c = 0; c < L.ncolors; ++c) {
        cl_sweep_list<false>(L, c, sw == 0 && c == 0, x, rhs, threadIdx.x, CLT);
        __syncthreads();
      }
  }
  for (int l = last - 1; l >= nd; --l) {
    const CLev& L = lev(l);
    const bool bin = l < nb;
    ClView V, W;
    if (bin) V = cl_view(C, l, 0, smem);
    if (l + 1 < nb) W = cl_view(C, l + 1, 0, smem);
    const int rows = bin ? V.nl : L.coff[L.ncolors - 1];  // every colour but the last
    for (int i = threadIdx.x; i < rows; i += CLT) {
      float xc;
      if (l + 1 < nb) {
        xc = cl_parent(V, W, i);
      } else {
        if (L.poff[i + 1] == L.poff[i]) continue;  // an empty bin
        xc = lx(l + 1)[L.pcol[L.poff[i]]];
      }
      float& x = bin ? V.x[V.B->plane + i] : lx(l)[i];
      x = __fadd_rn(x, __fmul_rn(C.alpha, xc));
    }
    __syncthreads();
    for (int sw = 0; sw < nu; ++sw)
      for (int c = bin ? 1 : L.ncolors - 1; c >= 0; --c) {
        if (bin) cl_sweep_smem(V, c, false, smem);
        else cl_sweep_list<false>(L, c, false, lx(l), lr(l), threadIdx.x, CLT);
        __syncthreads();
      }
  }
  // The first of these levels hands its iterate on through global memory.
  if (nd < nb) {
    const ClView V = cl_view(C, nd, 0, smem);
    for (int e = threadIdx.x; e < 2 * V.nl; e += CLT) {
      const int c = e >= V.nl ? 1 : 0, q = e - c * V.nl;
      V.B->gx[c * V.B->h + q] = V.x[c * V.ldx + V.B->plane + q];
    }
  } else {
    const CLev& L = lev(nd);
    for (int i = threadIdx.x; i < L.n; i += CLT) L.x[i] = lx(nd)[i];
  }
}

__global__ void __launch_bounds__(CLT, 1)
    k_coarse_cluster(const ClCase* cases, const CCase* cc, const MState* ST, int nu) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ClCase C;
  const int ci = blockIdx.x / CLS;
  if (!cases[ci].on || !active(ST, ci)) return;  // the whole cluster
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  {
    const long long* src = reinterpret_cast<const long long*>(&cases[ci]);
    long long* dst = reinterpret_cast<long long*>(&C);
    for (int w = threadIdx.x; w < (int)(sizeof(ClCase) / 8); w += CLT) dst[w] = src[w];
  }
  __syncthreads();
  const int nd = C.nd;
  // What stays for the whole cycle: zeroed iterates (halos included), row types, tables.
  for (int l = 0; l < C.nb; ++l) {
    if (l >= nd && rank != 0) break;
    const ClBin& B = C.b[l];
    const ClView V = cl_view(C, l, rank, smem);
    for (int e = threadIdx.x; e < 2 * V.ldx; e += CLT) V.x[e] = 0.0f;
    const int rows = B.layers * B.plane, at = V.k0 * B.plane;
    float4* t = reinterpret_cast<float4*>(smem + B.tab);
    for (int e = threadIdx.x; e < 3 * B.ntypes; e += CLT) t[e] = __ldg(&B.gtab[e]);
    if (B.type >= 0) {
      unsigned short* ty = reinterpret_cast<unsigned short*>(smem + B.type);
      for (int q = threadIdx.x; q < V.nl; q += CLT) {
        ty[q] = __ldg(&B.gtype[at + q]);
        ty[rows + q] = __ldg(&B.gtype[B.h + at + q]);
      }
    }
    if (l == 0 && nd > 0 && B.rhs >= 0) {
      float* rhs = reinterpret_cast<float*>(smem + B.rhs);
      for (int q = threadIdx.x; q < V.nl; q += CLT) {
        rhs[q] = __ldcg(&B.grhs[at + q]);
        rhs[rows + q] = __ldcg(&B.grhs[B.h + at + q]);
      }
    }
  }
  const CCase& D = cc[ci];
  const int tid = rank * CLT + threadIdx.x, nth = CLS * CLT;
  if (nd + C.ndl == 0) {  // small enough for one block
    __syncthreads();
    if (rank == 0) cl_first_block(C, D, nu, smem);
    return;
  }
  ClView V0{};
  if (nd > 0) V0 = cl_view(C, 0, rank, smem);
  const bool reg = nd > 0 && V0.B->rhs < 0;
  const float4* tab0 = nd > 0 ? reinterpret_cast<const float4*>(smem + V0.B->tab) : nullptr;
  ClRegs R;
  if (reg) {
    const int at = V0.k0 * V0.B->plane, h = V0.B->h;
#pragma unroll
    for (int m = 0; m < CLR; ++m) {
      const int q = threadIdx.x + m * CLT;
      if (q >= V0.nl) break;
      const unsigned t0 = __ldg(&V0.B->gtype[at + q]), t1 = __ldg(&V0.B->gtype[h + at + q]);
      R.type[0][m / 2] = m & 1 ? R.type[0][m / 2] | t0 << 16 : t0;
      R.type[1][m / 2] = m & 1 ? R.type[1][m / 2] | t1 << 16 : t1;
      R.rhs[0][m] = __ldcg(&V0.B->grhs[at + q]);
      R.rhs[1][m] = __ldcg(&V0.B->grhs[h + at + q]);
    }
  }
  cl.sync();
  // Down.
  for (int l = 0; l < nd; ++l) {
    const ClView V = l == 0 ? V0 : cl_view(C, l, rank, smem);
    const bool r0 = reg && l == 0;
    for (int sw = 0; sw < nu; ++sw) {
      if (r0) {
        if (sw == 0) cl_sweep_reg<0, true>(V, R, tab0);
        else cl_sweep_reg<0, false>(V, R, tab0);
        cl.sync();
        cl_sweep_reg<1, false>(V, R, tab0);
      } else {
        cl_sweep_smem(V, 0, sw == 0, smem);
        cl.sync();
        cl_sweep_smem(V, 1, false, smem);
      }
      cl.sync();
    }
    if (r0) {
      cl_resid_reg(V, R, tab0);
      __syncthreads();
    }
    if (l + 1 < nd) {
      const ClView W = cl_view(C, l + 1, rank, smem);
      const ClBin &B = *V.B, &N = *W.B;
      float* rhs = reinterpret_cast<float*>(smem + N.rhs);
      const int rows = N.layers * N.plane;
      for (int e = threadIdx.x; e < 2 * W.nl; e += CLT) {
        const int c = e >= W.nl ? 1 : 0, q = e - c * W.nl;
        const unsigned short* ty = reinterpret_cast<const unsigned short*>(smem + N.type);
        const int order = __float_as_int(reinterpret_cast<const float4*>(smem + N.tab)[3 * ty[c * rows + q] + 2].w);
        rhs[c * rows + q] = cl_restrict(W, c, q, order, B.nby, B.nbz, B.nbh, [&](int k, int j, int s) {
          const int f = (k - V.k0) * B.plane + j * B.nbh + s;
          return r0 ? V.x[B.plane + f] : cl_resid_smem(V, f, smem);
        });
      }
      __syncthreads();
    } else {
      float* res = V.B->gres + V.k0 * V.B->plane;
      for (int q = threadIdx.x; q < V.nl; q += CLT) res[q] = r0 ? V.x[V.B->plane + q] : cl_resid_smem(V, q, smem);
    }
  }
  cl.sync();
  for (int l = nd; l < nd + C.ndl; ++l) {  // split by rows: right-hand side, sweeps
    const CLev& L = D.lv[C.lc + l];
    if (l > 0) {
      const CLev& M = D.lv[C.lc + l - 1];
      for (int i = tid; i < L.n; i += nth) {
        float v = 0.0f;
        for (int k = M.roff[i]; k < M.roff[i + 1]; ++k) {
          const int ch = M.rchild[k];
          v = v + (l > nd ? cl_resid_list<true>(M, ch, M.x, M.rhs) : __ldcg(&M.res[ch]));
        }
        L.rhs[i] = v;
      }
      cl.sync();
    }
    for (int sw = 0; sw < nu; ++sw)
      for (int c = 0; c < L.ncolors; ++c) {
        cl_sweep_list<true>(L, c, sw == 0 && c == 0, L.x, L.rhs, tid, nth);
        cl.sync();
      }
  }
  if (rank == 0) cl_first_block(C, D, nu, smem);
  cl.sync();
  // Up.
  for (int l = nd + C.ndl - 1; l >= nd; --l) {
    const CLev &L = D.lv[C.lc + l], &N = D.lv[C.lc + l + 1];
    const int rows = L.coff[L.ncolors - 1];  // every colour but the last
    for (int i = tid; i < rows; i += nth) {
      const int p = L.poff[i];
      if (L.poff[i + 1] == p) continue;
      L.x[i] = __fadd_rn(__ldcg(&L.x[i]), __fmul_rn(C.alpha, __ldcg(&N.x[L.pcol[p]])));
    }
    cl.sync();
    for (int sw = 0; sw < nu; ++sw)
      for (int c = L.ncolors - 1; c >= 0; --c) {
        cl_sweep_list<true>(L, c, false, L.x, L.rhs, tid, nth);
        cl.sync();
      }
  }
  for (int l = nd - 1; l >= 0; --l) {
    const ClView V = l == 0 ? V0 : cl_view(C, l, rank, smem);
    const bool r0 = reg && l == 0;
    ClView W;
    if (l + 1 < nd) W = cl_view(C, l + 1, rank, smem);
    const CLev& L = D.lv[C.lc + l];
    const int at = V.k0 * V.B->plane;
    auto corr = [&](int q) {
      if (l + 1 < nd) return cl_parent(V, W, q);
      if (l + 1 < C.nb) return cl_parent_global(V, C.b[l + 1], q);
      const int p = L.poff[at + q];
      return L.poff[at + q + 1] == p ? 0.0f : __ldcg(&D.lv[C.lc + l + 1].x[L.pcol[p]]);
    };
    if (r0) {
#pragma unroll
      for (int m = 0; m < CLR; ++m) {
        const int q = threadIdx.x + m * CLT;
        if (q >= V.nl) break;
        cl_store(V, 0, q, __fadd_rn(R.keep[m], __fmul_rn(C.alpha, corr(q))));
      }
    } else {
      for (int q = threadIdx.x; q < V.nl; q += CLT)
        cl_store(V, 0, q, __fadd_rn(V.x[V.B->plane + q], __fmul_rn(C.alpha, corr(q))));
    }
    cl.sync();
    for (int sw = 0; sw < nu; ++sw) {
      if (r0) {
        cl_sweep_reg<1, false>(V, R, tab0);
        cl.sync();
        cl_sweep_reg<0, false>(V, R, tab0);
      } else {
        cl_sweep_smem(V, 1, false, smem);
        cl.sync();
        cl_sweep_smem(V, 0, false, smem);
      }
      cl.sync();
    }
  }
  pdl_leave();
  // The first level's iterate for the level above (the last cluster barrier also keeps every
  // block's shared memory alive until the stores into it have arrived).
  if (nd > 0) {
    const int at = V0.k0 * V0.B->plane;
    for (int e = threadIdx.x; e < 2 * V0.nl; e += CLT) {
      const int c = e >= V0.nl ? 1 : 0, q = e - c * V0.nl;
      V0.B->gx[c * V0.B->h + at + q] = V0.x[c * V0.ldx + V0.B->plane + q];
    }
  }
}

// ------------------------------------------------------------ levels above the clusters
// One launch a phase over every case (blockIdx.y), UPR rows a thread. The row types make a row
// 14 bytes of traffic (right-hand side, type, own and other colour) where its index list has
// about 70, and a launch that follows the one before closely costs less than the grid barrier
// and work search of the cooperative phases: the coarse levels of 8.4 M cells (1,048,576 rows on
// the first) 206 -> 136 us, of 160x160x80 cells 166 -> 99 us, the projections 11.97 -> 10.81 ms
// and, of eight uneven cases, 7.53 -> 6.73 ms.
constexpr int UPT = 256, UPR = 2;

template <int C, bool FIRST>
__global__ void __launch_bounds__(UPT) k_up_sweep(const ClUp* ups, const MState* ST, int l) {
  pdl_enter();
  const ClUp& U = ups[blockIdx.y];
  if (l >= U.n || !active(ST, blockIdx.y)) return;
  const ClBin& B = U.lv[l];
  const int h = B.h;
  const float* __restrict__ xo = B.gx + (1 - C) * h;
  unsigned type[UPR];
  float v[UPR];
#pragma unroll
  for (int m = 0; m < UPR; ++m) {
    const int q = (blockIdx.x * UPR + m) * UPT + threadIdx.x;
    type[m] = q < h ? __ldg(&B.gtype[C * h + q]) : 0;
    v[m] = q < h ? B.grhs[C * h + q] : 0.0f;
  }
#pragma unroll
  for (int m = 0; m < UPR; ++m) {
    const int q = (blockIdx.x * UPR + m) * UPT + threadIdx.x;
    if (q >= h) break;
    const float4 *t = B.gtab + 3 * type[m], b = __ldg(t + 1);
    if (!FIRST) {
      ClRow r;
      r.a = __ldg(t);
      r.b = b;
      r.o = __ldg(reinterpret_cast<const int4*>(t + 2));
      v[m] = cl_sum<true>(v[m], xo + q, r);
    }
    B.gx[C * h + q] = v[m] * b.w;
  }
}

// The next level's right-hand side from the colour-0 residuals of its children.
__global__ void __launch_bounds__(UPT) k_up_restrict(const ClUp* ups, const MState* ST, int l) {
  pdl_enter();
  const ClUp& U = ups[blockIdx.y];
  if (l >= U.n || !active(ST, blockIdx.y)) return;
  const ClBin &B = U.lv[l], &N = U.lv[l + 1];
  const int e = blockIdx.x * UPT + threadIdx.x;
  if (e >= 2 * N.h) return;
  const int c = e >= N.h ? 1 : 0, q = e - c * N.h;
  ClView W;
  W.B = &N;
  W.k0 = 0;
  const int order = __float_as_int(__ldg(&N.gtab[3 * __ldg(&N.gtype[e]) + 2].w));
  U.rhs[l + 1][e] = cl_restrict(W, c, q, order, B.nby, B.nbz, B.nbh, [&](int k, int j, int s) {
    const int f = (k * B.nby + j) * B.nbh + s;
    const float4* t = B.gtab + 3 * __ldg(&B.gtype[f]);
    ClRow r;
    r.a = __ldg(t);
    r.b = __ldg(t + 1);
    r.o = __ldg(reinterpret_cast<const int4*>(t + 2));
    return B.grhs[f] - cl_sum<false>(__fmul_rn(r.b.z, B.gx[f]), B.gx + B.h + f, r);
  });
}

// Colour 0 takes its correction (colour 1 is swept next without being read).
__global__ void __launch_bounds__(UPT) k_up_prolong(const ClUp* ups, const MState* ST, int l) {
  pdl_enter();
  const ClUp& U = ups[blockIdx.y];
  if (l >= U.n || !active(ST, blockIdx.y)) return;
  const ClBin &B = U.lv[l], &N = U.lv[l + 1];
  const int q = blockIdx.x * UPT + threadIdx.x;
  if (q >= B.h) return;
  ClView V;
  V.B = &B;
  V.k0 = 0;
  B.gx[q] = __fadd_rn(B.gx[q], __fmul_rn(U.alpha, cl_parent_global(V, N, q)));
}
