// Where the threads of a wavefront sweep (wave.cuh) read: the tiles, a compute thread's
// pencil and the indices of the neighbours it loads. Plain C++ as well as device code, so
// that a host test can walk every thread of every tile.
#pragma once

#ifdef __CUDACC__
#define CFDG_HD __host__ __device__ __forceinline__
#else
#define CFDG_HD inline
#endif

namespace cfdg {

constexpr int WTJ = 8, WTK = 8;       // tile of pencils per CTA
constexpr int WCT = WTJ * WTK;        // compute threads (two warps)
constexpr int WRING = 256;            // received values per boundary pencil held in shared memory
constexpr int WHALO = WTJ + WTK;      // boundary pencils of a tile that its consumers read
constexpr int WSHARED = 2 * WCT + WHALO * WRING;  // the last two steps' values, [step & 1][thread]; the ring, [pencil][WRING]

enum WaveMode { IC0_FWD = 0, IC0_BWD = 1, GS_FWD = 2, GS_BWD = 3 };

// Hand-off entries: the boundary pencils between tiles that follow one another along j, [K][J][step
// along x][k in the tile], then those along k, [K][J][step along x][j in the tile]; J, K the lower
// tile of the two. A sweep either way uses the same ones.
CFDG_HD long long wave_halo_y(int J, int K, int nx, int tiles_j) { return ((long long)K * (tiles_j - 1) + J) * nx * WTK; }
CFDG_HD long long wave_halo_z(int J, int K, int nx, int tiles_j, int tiles_k) {
  return (long long)tiles_k * (tiles_j - 1) * nx * WTK + ((long long)K * tiles_j + J) * nx * WTJ;
}
CFDG_HD long long wave_halo_size(int nx, int tiles_j, int tiles_k) { return wave_halo_z(0, tiles_k - 1, nx, tiles_j, tiles_k); }

template <int MODE>
struct WavePlace {
  static constexpr bool BWD = MODE == IC0_BWD || MODE == GS_BWD;
  static constexpr int dir = BWD ? -1 : 1;
  int tj, tk, j, k;
  bool on;   // the thread owns a pencil
  int row;   // the pencil's first cell (structured grids have fewer than 2^31 cells)
  int dj, dk;  // distance of the pencil from the tile's first one in sweep order
  bool edge_y, edge_z;  // the new values along j, k come from the tile before this one
  int oy, oz;           // offsets of the neighbours along j and k that are loaded ahead
  int near_y, near_z;   // threads whose last values are the new ones along j and k, inside the tile

  // A thread without a pencil goes through the motions on the first one with its own entries in
  // place of every neighbour: whether there is a neighbour is asked only for a pencil's own
  // thread, and nothing outside the arrays is read.
  CFDG_HD WavePlace(int tid, int J, int K, int nx, int ny, int nz) {
    tj = tid % WTJ, tk = tid / WTJ;
    j = J * WTJ + tj, k = K * WTK + tk;
    on = j < ny && k < nz;
    row = on ? (k * ny + j) * nx : 0;
    dj = BWD ? WTJ - 1 - tj : tj, dk = BWD ? WTK - 1 - tk : tk;
    const bool has_ny = on && (BWD ? j + 1 < ny : j > 0), has_nz = on && (BWD ? k + 1 < nz : k > 0);
    edge_y = dj == 0 && has_ny, edge_z = dk == 0 && has_nz;
    // IC(0) backward reads the new neighbours' coefficients, Gauss-Seidel the values not updated
    // yet. Where there is none the cell's own entry stands in, unused.
    const bool has_oy = MODE == IC0_BWD ? has_ny : on && (BWD ? j > 0 : j + 1 < ny);
    const bool has_oz = MODE == IC0_BWD ? has_nz : on && (BWD ? k > 0 : k + 1 < nz);
    oy = has_oy ? (MODE == IC0_BWD ? nx : dir * nx) : 0;
    oz = has_oz ? (MODE == IC0_BWD ? nx * ny : dir * nx * ny) : 0;
    near_y = has_ny && !edge_y ? tid - dir : tid;
    near_z = has_nz && !edge_z ? tid - dir * WTJ : tid;
  }
  // The cell at place `at` (0 .. nx-1) of the sweep along the pencil, and the offset of its
  // neighbour along x that is loaded ahead (its own entry where there is none).
  CFDG_HD int cell(int at, int nx) const { return row + (BWD ? nx - 1 - at : at); }
  static CFDG_HD int ox(int at, int nx) {
    return MODE == IC0_BWD ? (at > 0 ? 1 : 0) : (at + 1 < nx ? dir : 0);
  }
  // Where the new values that the tile before this one along j (k) hands over start, this one's
  // lane first, and where this pencil's go to the tile behind it; the values of a pencil follow
  // one another WTK (WTJ) entries apart. Only for tiles that have one before, behind.
  static CFDG_HD long long from_y(int J, int K, int nx, int tiles_j) { return wave_halo_y(BWD ? J : J - 1, K, nx, tiles_j); }
  static CFDG_HD long long from_z(int J, int K, int nx, int tiles_j, int tiles_k) {
    return wave_halo_z(J, BWD ? K : K - 1, nx, tiles_j, tiles_k);
  }
  CFDG_HD long long to_y(int J, int K, int nx, int tiles_j) const { return wave_halo_y(BWD ? J - 1 : J, K, nx, tiles_j) + tk; }
  CFDG_HD long long to_z(int J, int K, int nx, int tiles_j, int tiles_k) const {
    return wave_halo_z(J, BWD ? K - 1 : K, nx, tiles_j, tiles_k) + tj;
  }
  // Places in the shared array of the new values along j and k; `at` is any number.
  CFDG_HD int new_y(int at, int before) const {
    return edge_y ? 2 * WCT + tk * WRING + (at & (WRING - 1)) : before + near_y;
  }
  CFDG_HD int new_z(int at, int before) const {
    return edge_z ? 2 * WCT + (WTK + tj) * WRING + (at & (WRING - 1)) : before + near_z;
  }
};

}  // namespace cfdg
