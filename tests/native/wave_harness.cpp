// Test harness (tests only): walks every compute thread of every tile of a wavefront sweep
// (cfd-craft_gb300/csrc/wave_place.hpp, the arithmetic that the kernel runs) over all places of
// its pencil and counts the reads outside the arrays and the neighbours that are not the cell's.
#include <cstdint>
#include <vector>

#include "wave_place.hpp"

using namespace cfdg;

// The hand-off entries: every value goes where the tile behind reads it, none is shared.
template <int MODE>
static void halo(int nx, int ny, int nz, int64_t* out) {
  using P = WavePlace<MODE>;
  const int tj = (ny + WTJ - 1) / WTJ, tk = (nz + WTK - 1) / WTK, s = P::dir;
  std::vector<int> used(wave_halo_size(nx, tj, tk), 0);
  for (int K = 0; K < tk; ++K)
    for (int J = 0; J < tj; ++J)
      for (int tid = 0; tid < WCT; ++tid) {
        const P p(tid, J, K, nx, ny, nz);
        if (!p.on) continue;
        for (int way = 0; way < 2; ++way) {
          const int J2 = way ? J : J + s, K2 = way ? K + s : K, d = way ? p.dk : p.dj;
          if (d != WTJ - 1 || J2 < 0 || J2 >= tj || K2 < 0 || K2 >= tk) continue;
          const long long to = way ? p.to_z(J, K, nx, tj, tk) : p.to_y(J, K, nx, tj);
          const long long from =
              way ? P::from_z(J2, K2, nx, tj, tk) + p.tj : P::from_y(J2, K2, nx, tj) + p.tk;
          if (to != from) ++out[2];
          for (int at = 0; at < nx; ++at) {
            const long long e = to + (long long)at * WTK;
            if (e < 0 || e >= (long long)used.size() || used[e]++) ++out[0];
          }
        }
      }
}

template <int MODE>
static void scan(int nx, int ny, int nz, int64_t* out) {
  using P = WavePlace<MODE>;
  const int64_t N = (int64_t)nx * ny * nz;
  const int s = P::dir;
  for (int K = 0; K < (nz + WTK - 1) / WTK; ++K)
    for (int J = 0; J < (ny + WTJ - 1) / WTJ; ++J)
      for (int tid = 0; tid < WCT; ++tid) {
        const P p(tid, J, K, nx, ny, nz);
        const int last = nx + 2 * (WTJ + WTK);
        for (int step = -(WTJ + WTK); step < last; ++step) {
          const int at = step < 0 ? 0 : step < nx ? step : nx - 1;
          const int64_t c = p.cell(at, nx), o[3] = {c + P::ox(at, nx), c + p.oy, c + p.oz};
          if (c < 0 || c >= N) ++out[0];
          for (int a = 0; a < 3; ++a)
            if (o[a] < 0 || o[a] >= N) ++out[0];
          for (int before = 0; before <= WCT; before += WCT) {
            const int y = p.new_y(step, before), z = p.new_z(step, before);
            if (y < 0 || y >= WSHARED || z < 0 || z >= WSHARED) ++out[1];
            // Inside the step's values or the ring, not across their border.
            if ((y < 2 * WCT) != !p.edge_y || (z < 2 * WCT) != !p.edge_z) ++out[1];
            if (!p.edge_y && (y < before || y >= before + WCT)) ++out[1];
            if (!p.edge_z && (z < before || z >= before + WCT)) ++out[1];
          }
          if (!p.on) continue;
          ++out[3];
          // The neighbour loaded ahead: IC(0) backward the one updated before, Gauss-Seidel the
          // one updated after; the new value along j or k: the one updated before.
          const int i = P::BWD ? nx - 1 - at : at, d = MODE == IC0_BWD ? 1 : s;
          const int q[3] = {i, p.j, p.k}, n[3] = {nx, ny, nz};
          const int64_t stride[3] = {1, nx, (int64_t)nx * ny};
          if (c != i + nx * (p.j + (int64_t)ny * p.k)) ++out[2];
          for (int a = 0; a < 3; ++a) {
            const bool has = q[a] + d >= 0 && q[a] + d < n[a];
            if (o[a] != c + (has ? d * stride[a] : 0)) ++out[2];
          }
          const bool ny_ = p.j - s >= 0 && p.j - s < ny, nz_ = p.k - s >= 0 && p.k - s < nz;
          const bool in_y = ny_ && (p.j - s) / WTJ == J, in_z = nz_ && (p.k - s) / WTK == K;
          if (p.edge_y != (ny_ && !in_y) || p.edge_z != (nz_ && !in_z)) ++out[2];
          if (in_y && p.new_y(step, 0) != p.tk * WTJ + p.tj - s) ++out[2];
          if (in_z && p.new_z(step, 0) != (p.tk - s) * WTJ + p.tj) ++out[2];
        }
      }
}

// out: reads (and hand-off entries) outside the arrays, reads outside the shared array or its parts, wrong neighbours,
// cells visited by their own threads (with the clamped steps).
extern "C" void wave_scan(int mode, int nx, int ny, int nz, int64_t* out) {
  for (int a = 0; a < 4; ++a) out[a] = 0;
  if (mode == IC0_FWD) scan<IC0_FWD>(nx, ny, nz, out), halo<IC0_FWD>(nx, ny, nz, out);
  if (mode == IC0_BWD) scan<IC0_BWD>(nx, ny, nz, out), halo<IC0_BWD>(nx, ny, nz, out);
  if (mode == GS_FWD) scan<GS_FWD>(nx, ny, nz, out), halo<GS_FWD>(nx, ny, nz, out);
  if (mode == GS_BWD) scan<GS_BWD>(nx, ny, nz, out), halo<GS_BWD>(nx, ny, nz, out);
}
