// Pipelined wavefront sweeps over the structured fine level (one launch per sweep).
//
// A lexicographic sweep over the 7-point pattern in natural cell order (IC(0)
// forward/backward substitution, pressure.rs:225-240; Gauss-Seidel,
// multigrid.rs:272-281 / masked.rs:158-172) updates cell (i,j,k) after (i-1,j,k),
// (i,j-1,k) and (i,j,k-1). Each CTA owns a TJ x TK tile of x-pencils; compute thread
// (tj,tk) walks its pencil and handles cell i at local step s = i + tj + tk, so the cells
// of one step lie on a hyperplane of the tile. Values of the previous step come from
// shared memory (one barrier of the two compute warps per step), the pencil's own
// predecessor from a register. Tiles depend on their (J-1,K) and (J,K-1) neighbours only
// through the boundary pencils: a boundary thread stores each new value together with the
// launch's epoch in one 16-byte store, and a receiver warp of the consuming tile polls
// those entries (four per lane and round trip, bounded) into a shared ring, so the compute
// threads never wait on global memory but for data not produced yet. Tiles are taken in a
// topological order from an atomic ticket, so a CTA only ever waits for tiles already held
// by running CTAs; the ticket counts on from launch to launch and gives the epoch, so
// nothing is cleared between launches.
//
// Bound: the instructions of one warp's step, nx + ny + nz of them in a row plus a hand-off
// of about a microsecond per tile on the way. A warp's FP64 operation takes 64 cycles on
// this part (31 ns, measured; independent ones of the same warp do not overlap), so a
// Gauss-Seidel step's fifteen (six sums, six products, three of the division) cost at least
// 0.46 us. What else a step does is kept off that chain and free of branches: the operands
// that do not depend on the sweep (right-hand side, flags, diagonal, the neighbours not
// updated yet) are loaded WPF steps ahead into registers, absent faces are selected to a
// neutral zero, and the correctly rounded division by the diagonal uses its precomputed
// reciprocal (div_pre: three or five operations instead of 272 ns). One Gauss-Seidel sweep
// of 128x128x64 takes 275 us, of 64x64x32 136 us; with a flag poll, a fence, unprefetched
// loads, branches and a division per step the former took 1295 us. An IC(0) application
// (both sweeps) of 64x64x32 takes 242 us (954 us). Tiles of one warp (8 x 4) gave 310 us.
//
// Every cell is computed with the same operations in the same order as the
// reference's natural-order loop, so the result is bit-identical to it. Backward
// sweeps run the same machinery mirrored (i, j, k descending).
#pragma once
#include "plain_kernels.cuh"
#include "wave_place.hpp"

namespace cfdg {

constexpr int WTHREADS = WCT + 32;    // the compute threads and the receiver warp
constexpr int WPF = 4;                // steps of operands in flight per compute thread

struct WaveArgs {
  int n[3];
  int tiles_j, tiles_k;
  const uint16_t* flags;  // interior/outlet face bits per cell (GridDev::flags layout)
  const double* in;       // r (IC0_FWD) or rhs (GS_*)
  double* x;              // z (IC0_*; IC0_BWD in place) or x (GS_*, in place)
  const double* diag;     // IC(0) factor diagonal, or the level-0 matrix diagonal
  const double* rdiag;    // its reciprocals as div_pre takes them (k_recip)
  const double* lx;       // IC(0): lower coefficient of each row towards (i-1), (j-1), (k-1)
  const double* ly;
  const double* lz;
  // Gauss-Seidel weights: uniform per axis, or per face.
  double w_in[3];
  const double* fw;
  long long face_off[3];
  int fdim[3][3];
  unsigned long long* sync;  // [0] tickets taken so far, [1] epoch of the last launch that gave up
  ulonglong2* halo;          // boundary values (wave_halo_y, wave_halo_z): their bits and epoch
  int* error;                // persistent: set to 1 when a wait gave up
  const Scalars* S;
  long long spin_limit;  // polls before a wait gives up (WAVE_SPIN_LIMIT)
  int hold_tile;         // -1; a test of the bounded waits names a tile that never publishes
};

// One 16-byte access each way (PTX b128): the value and its epoch arrive together.
__device__ __forceinline__ void st_halo(ulonglong2* p, double v, unsigned long long epoch, bool on) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.b128 t, {%1, %2};\n\t"
      "@p st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"((unsigned long long)__double_as_longlong(v)), "l"(epoch), "r"((unsigned)on)
      : "memory");
}
__device__ __forceinline__ ulonglong2 ld_halo(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// The division by a known divisor. rd is recip_of(d): r = RN(1/d), negative where the first
// quotient below may be more than one ulp off, 0 where d lies outside [2^-60, 2^60].
__device__ __forceinline__ double recip_of(double d) {
  if (!(d >= 0x1p-60 && d <= 0x1p60)) return 0.0;
  const double r = __drcp_rn(d);
  return fabs(__fma_rn(r, d, -1.0)) <= 0x1p-54 ? r : -r;
}
__device__ __noinline__ double div_rare(double v, double d) { return __ddiv_rn(v, d); }

// v / d, correctly rounded, by Markstein's correction step (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990): from r = RN(1/d) and q within one ulp of v/d, the remainder v - q d is
// exact under one FMA and RN(q + rem r) is RN(v/d). q = RN(v r) is within one ulp when
// |r d - 1| <= 2^-54: with significands v, d in [1, 2) its error is at most v |r - 1/d|
// plus half an ulp of q, v |r - 1/d| <= 2^-54 v/d, and v/d < 1 halves the ulp, so both
// cases stay within one ulp. Otherwise (rd < 0) one more correction first makes it so.
// A zero is its own quotient (solid cells, and cells that nothing has reached yet: with a
// division for them an IC(0) iteration of 24x20x16 took 157 us instead of 115). Subnormals,
// NaN, infinities and other v outside [2^-900, 2^900] (where a product or remainder could
// leave the normal range) take the division. The tests are on the bits: a
// comparison of doubles would queue for the FP64 pipe. on: whether the result is used;
// EXTRA: whether some rd is negative (a warp's FP64 operations take 64 cycles each, also
// where no lane needs them).
template <bool EXTRA>
__device__ __forceinline__ double div_pre(double v, double d, double rd, bool on) {
  const int hi = __double2hiint(rd);
  const double r = fabs(rd);
  double q = __dmul_rn(v, r);
  double rem = __fma_rn(-q, d, v);
  q = __fma_rn(rem, r, q);
  if (EXTRA && hi < 0) {
    rem = __fma_rn(-q, d, v);
    q = __fma_rn(rem, r, q);
  }
  const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
  if (on && (e - 123u > 1800u || hi == 0)) {
    const unsigned mag = (unsigned)__double2hiint(v) << 1 | (unsigned)__double2loint(v);
    if (mag == 0 && hi != 0) q = v;
    else q = div_rare(v, d);
  }
  return q;
}

// rd = recip_of(d) for n divisors; *extra is set when one of them is negative.
__global__ void k_recip(const double* __restrict__ d, double* __restrict__ rd, long long n, int* extra) {
  bool neg = false;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double r = recip_of(d[i]);
    rd[i] = r;
    neg |= r < 0.0;
  }
  if (neg) *extra = 1;
}

// The operands of one cell that do not depend on the sweep.
template <int MODE, bool UNIFORM>
struct WaveCell {
  unsigned fl;
  double in, d, rd;
  double o[3];                                     // GS: the neighbours not updated yet; IC(0): the coefficients
  double w[(MODE >= GS_FWD && !UNIFORM) ? 6 : 1];  // GS on non-uniform grids: the face weights
};

template <int MODE, bool UNIFORM, bool EXTRA>
__global__ void __launch_bounds__(WTHREADS) k_wave(WaveArgs A) {
  constexpr bool BWD = (MODE == IC0_BWD || MODE == GS_BWD);
  constexpr bool GS = MODE >= GS_FWD;
  __shared__ double sh[WSHARED];
  double* const ring = sh + 2 * WCT;
  __shared__ volatile int seen[WHALO];  // values received per boundary pencil
  __shared__ volatile int passed;       // steps whose barrier the compute warps have passed
  __shared__ volatile int bail;
  __shared__ unsigned long long ticket;
  pdl_enter();
  if (A.S && A.S->done) return;
  const int nx = A.n[0], ny = A.n[1], nz = A.n[2];
  if (threadIdx.x == 0) {
    ticket = atomicAdd(&A.sync[0], 1ull);
    passed = 0;
    bail = 0;
  }
  if (threadIdx.x < WHALO) seen[threadIdx.x] = 0;
  __syncthreads();
  const unsigned ntiles = gridDim.x;  // every block of every launch takes one ticket
  const unsigned long long epoch = ticket / ntiles + 1;
  const int t = (int)(ticket % ntiles);
  int J = t % A.tiles_j, K = t / A.tiles_j;  // row-major tiles: producers have smaller tickets
  if (BWD) {
    J = A.tiles_j - 1 - J;
    K = A.tiles_k - 1 - K;
  }
  if (threadIdx.x >= WCT) {
    // Receiver warp: lane p < WTJ + WTK follows one boundary pencil of the tile before this
    // one along j (lanes 0 .. WTK-1: its last pencil column, one per k) or along k. All lanes
    // take every turn of the loop together, so one round trip serves them all.
    const int lane = threadIdx.x - WCT;
    const bool along_j = lane < WTK;
    const int p = along_j ? lane : lane - WTK;
    bool open = lane < WHALO && (along_j ? (BWD ? J + 1 < A.tiles_j : J > 0) && K * WTK + p < nz
                                         : (BWD ? K + 1 < A.tiles_k : K > 0) && J * WTJ + p < ny);
    const ulonglong2* src = A.halo;
    if (open)
      src += p + (along_j ? WavePlace<MODE>::from_y(J, K, nx, A.tiles_j)
                          : WavePlace<MODE>::from_z(J, K, nx, A.tiles_j, A.tiles_k));
    // The pencil's first cell is used at step `late`: entries below passed - late are free.
    const int late = BWD ? (along_j ? WTK : WTJ) - 1 - p : p;
    int got = 0;
    long long polls = 0;
    for (unsigned turn = 1; __any_sync(0xffffffffu, open); ++turn) {
      const bool room = open && got + 4 <= passed - late + WRING;
      int m = 0;
      if (room) {
        ulonglong2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = ld_halo(src + (long long)min(got + q, nx - 1) * WTK);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (m == q && got + q < nx && v[q].y == epoch) {
            ring[lane * WRING + ((got + q) & (WRING - 1))] = __longlong_as_double((long long)v[q].x);
            m = q + 1;
          }
        if (m) {
          got += m;
          __threadfence_block();
          seen[lane] = got;
          open = got < nx;
        }
        polls = m ? 0 : polls + 1;
      }
      const bool late_launch = (turn & 63u) == 0 && ld_relaxed(&A.sync[1]) == epoch;
      if (__any_sync(0xffffffffu, polls > A.spin_limit || late_launch)) {
        // Give up: flag the launch and let the compute warps run out without waiting; the
        // host discards the result.
        if (lane == 0) {
          atomicExch(&A.sync[1], epoch);
          atomicExch(A.error, 1);
          bail = 1;
        }
        return;
      }
    }
    return;
  }
  // A thread without a pencil goes through the motions on the first one (WavePlace); its values
  // are not stored, published or read by any other cell.
  const WavePlace<MODE> P((int)threadIdx.x, J, K, nx, ny, nz);
  const int tj = P.tj, tk = P.tk;
  const int len = P.on ? nx : 0;  // cells of this thread's pencil
  constexpr int dir = BWD ? -1 : 1;
  const int nsteps = nx + WTJ + WTK - 2;
  const bool pub_y = P.on && P.dj == WTJ - 1 && (BWD ? J > 0 : J + 1 < A.tiles_j) && t != A.hold_tile;
  const bool pub_z = P.on && P.dk == WTK - 1 && (BWD ? K > 0 : K + 1 < A.tiles_k) && t != A.hold_tile;
  // Entries (fewer than half the cells) that this pencil's next values go to.
  int to_y = (pub_y ? (int)P.to_y(J, K, nx, A.tiles_j) : 0) - (P.dj + P.dk) * WTK;
  int to_z = (pub_z ? (int)P.to_z(J, K, nx, A.tiles_j, A.tiles_k) : 0) - (P.dj + P.dk) * WTJ;
  using Cell = WaveCell<MODE, UNIFORM>;
  Cell cell[WPF];
  int fat = -P.dj - P.dk;  // the cell (in sweep order) fetched next
  // No branch: outside the pencil its end cell is fetched again, unused.
  auto fetch = [&](Cell& C) {
    const int at = min(max(fat, 0), nx - 1);
    const int c = P.cell(at, nx);
    C.fl = A.flags[c];
    C.d = A.diag[c];
    C.rd = A.rdiag[c];
    if (MODE == IC0_FWD) {
      C.in = A.in[c];
      C.o[0] = A.lx[c], C.o[1] = A.ly[c], C.o[2] = A.lz[c];
    } else if (MODE == IC0_BWD) {
      // Rows (k+1), (j+1), (i+1), each with its coefficient towards this cell.
      C.in = A.x[c];
      C.o[0] = A.lx[c + P.ox(at, nx)];
      C.o[1] = A.ly[c + P.oy];
      C.o[2] = A.lz[c + P.oz];
    } else {
      C.in = A.in[c];
      C.o[0] = A.x[c + P.ox(at, nx)];
      C.o[1] = A.x[c + P.oy];
      C.o[2] = A.x[c + P.oz];
      if (!UNIFORM) {
        const int q[3] = {BWD ? nx - 1 - at : at, P.on ? P.j : 0, P.on ? P.k : 0};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          int f[3] = {q[0], q[1], q[2]};
          C.w[2 * a] = A.fw[A.face_off[a] + ((long long)f[2] * A.fdim[a][1] + f[1]) * A.fdim[a][0] + f[0]];
          f[a] += 1;
          C.w[2 * a + 1] = A.fw[A.face_off[a] + ((long long)f[2] * A.fdim[a][1] + f[1]) * A.fdim[a][0] + f[0]];
        }
      }
    }
    ++fat;
  };
  // Face f of the cell, where it is in the operator: its weight (GS).
  const double w0 = A.w_in[0], w1 = A.w_in[1], w2 = A.w_in[2];
  auto weight = [&](const Cell& C, int f) {
    return UNIFORM ? (f < 2 ? w0 : f < 4 ? w1 : w2) : C.w[GS && !UNIFORM ? f : 0];
  };
  // A term of a row, or the zero whose sum (GS) or difference (IC(0)) leaves every number's
  // bits alone: -0.0 added, +0.0 subtracted. Selected, not branched around.
  auto term = [&](const Cell& C, int f, double w, double x) {
    const double p = w * x;
    return (C.fl & (1u << f)) ? p : (GS ? -0.0 : 0.0);
  };
  double old[3];  // GS: the terms of the neighbours not updated yet, of the step to come
  auto old_terms = [&](const Cell& C) {
    if (GS) {
#pragma unroll
      for (int a = 0; a < 3; ++a) old[a] = term(C, 2 * a + (BWD ? 0 : 1), weight(C, 2 * a + (BWD ? 0 : 1)), C.o[a]);
    }
  };
  double prev = 0.0;  // this pencil's value at the previous cell in sweep order
  int have_y = P.edge_y ? 0 : nx, have_z = P.edge_z ? 0 : nx;  // received values as last seen
#pragma unroll
  for (int m = 0; m < WPF; ++m) fetch(cell[m]);
  old_terms(cell[0]);
  int at = -P.dj - P.dk, c = P.row + (BWD ? nx - 1 : 0) + dir * at;
  for (int s0 = 0; s0 < nsteps; s0 += WPF) {  // steps past nsteps - 1 find no cell in range
#pragma unroll
    for (int m = 0; m < WPF; ++m, ++at, c += dir, to_y += WTK, to_z += WTJ) {
      Cell& C = cell[m];
      const bool on = (unsigned)at < (unsigned)len;
      while (__any_sync(0xffffffffu, on && (have_y <= at || have_z <= at))) {
        if (P.edge_y) have_y = seen[tk];
        if (P.edge_z) have_z = seen[WTK + tj];
        if (bail) have_y = have_z = nx;
      }
      // The step before is in sh. (The vote that ends the loop above has brought the warp together.)
      asm volatile("bar.sync 1, %0;" ::"n"(WCT) : "memory");
      if (m == 0 && threadIdx.x == 0) passed = s0;
      const int before = ((m + 1) & 1) * WCT;  // WPF is even: step parity is m's
      const double newy = sh[P.new_y(at, before)];
      const double newz = sh[P.new_z(at, before)];
      double v = C.in;
      if (MODE == IC0_FWD) {
        // Ascending columns: (k-1), (j-1), (i-1).
        v = v - term(C, 4, C.o[2], newz);
        v = v - term(C, 2, C.o[1], newy);
        v = v - term(C, 0, C.o[0], prev);
        v = div_pre<EXTRA>(v, C.d, C.rd, on);
      } else if (MODE == IC0_BWD) {
        // Rows (k+1), (j+1), (i+1) in descending order.
        v = v - term(C, 5, C.o[2], newz);
        v = v - term(C, 3, C.o[1], newy);
        v = v - term(C, 1, C.o[0], prev);
        v = div_pre<EXTRA>(v, C.d, C.rd, on);
      } else {
        // Row order x-lo, x-hi, y-lo, y-hi, z-lo, z-hi; entries are -w, and v - (-w) x == v + w x
        // exactly.
        const double nx_ = term(C, BWD ? 1 : 0, weight(C, BWD ? 1 : 0), prev);
        const double ny_ = term(C, BWD ? 3 : 2, weight(C, BWD ? 3 : 2), newy);
        const double nz_ = term(C, BWD ? 5 : 4, weight(C, BWD ? 5 : 4), newz);
        v = v + (BWD ? old[0] : nx_);
        v = v + (BWD ? nx_ : old[0]);
        v = v + (BWD ? old[1] : ny_);
        v = v + (BWD ? ny_ : old[1]);
        v = v + (BWD ? old[2] : nz_);
        v = v + (BWD ? nz_ : old[2]);
        // d = 0: a cell with no faces in the operator (a sealed singleton, or a solid cell).
        const bool some = ((unsigned)__double2hiint(C.d) << 1 | (unsigned)__double2loint(C.d)) != 0;
        v = div_pre<EXTRA>(v, C.d, C.rd, on && some);
        if (!some) v = 0.0;
      }
      sh[(m & 1) * WCT + threadIdx.x] = v;
      prev = v;
      st_halo(A.halo + to_y, v, epoch, on && pub_y);
      st_halo(A.halo + to_z, v, epoch, on && pub_z);
      if (on) A.x[c] = v;
      old_terms(cell[(m + 1) % WPF]);
      fetch(C);
    }
  }
}

static_assert(WTJ == WTK, "the receiver's lanes step alike along both boundaries");
static_assert(WPF % 2 == 0, "the step's buffer is chosen by its place in the unrolled group");

}  // namespace cfdg
