// Host check of the row-tile index arithmetic (gpu-sims_b200/csrc/phys_rows.cuh)
// against the node formulas of the esoteric-pull layout: for every node, the
// element each population is read from and written to, the bounds and the
// 16-byte rules of the copies, and that no two threads or tiles share an
// element.  Runs on the CPU.
#include <cstdio>
#include <random>
#include <utility>
#include <vector>

#include "../gpu-sims_b200/csrc/phys_rows.cuh"

using namespace lbm;

template <int PREC>
long check(int nx, int ny, int nz, const int (&per)[3]) {
  using T = typename Store<PREC>::T;
  constexpr uint32_t EB = sizeof(T);
  PhysGeom g{};
  g.nx = nx; g.ny = ny; g.nz = nz;
  g.n = (size_t)nx * ny * nz;
  for (int a = 0; a < 3; ++a) g.per[a] = per[a];
  g.px = (nx + (per[0] ? 0 : 1) + 7) / 8 * 8;
  g.gy = per[1] ? 0 : 1;
  g.gz = per[2] ? 0 : 1;
  g.py = ny + 2 * g.gy;
  g.pz = nz + 2 * g.gz;
  g.pxy = (uint32_t)(g.px * g.py);
  g.slot_stride = ((size_t)g.pxy * g.pz + 63) / 64 * 64;
  const size_t SS = g.slot_stride;
  const RowTiles rt = row_tiles(g);
  if (!rt.R) return 0;
  long bad = 0;
  char* base = (char*)(uintptr_t)0x100000000ull;  // never dereferenced
  const uint32_t rb = g.px * EB;
  for (int P = 0; P < 2; ++P) {
    std::vector<int> written(Q * SS, -1);
    for (uint32_t t = 0; t < rt.ntiles; ++t) {
      RowWalk w;  // tile t reached by strides of 7
      w.start(t % 7, 7, rt.tiles_y);
      for (uint32_t k = t % 7; k < t; k += 7) w.next(rt.tiles_y);
      const int z = w.z, y0 = w.ty * rt.R, rows = std::min(rt.R, ny - y0);
      bad += (uint32_t)(z * rt.tiles_y + w.ty) != t;
      // element of the store behind every 2 bytes of the stage
      std::vector<long> src(rows_stage<PREC>() / 2, -1), dst(rows_stage<PREC>() / 2, -1);
      const size_t at0 = lin(g, 0, y0, z);
      const bool inner = y0 > 0 && y0 + rows < ny && z > 0 && z < nz - 1;
      for (int k = 0; k < Q; ++k)
        for (int load = 1; load >= 0; --load) {
          int total = 0;
          auto copy = [&](ptrdiff_t rel, int r, int cnt) {
            const size_t el = at0 + rel;
            const uint32_t so = k * rows_region<PREC>() + r * rb;
            total += cnt;
            bad += inner && (rel != array_offset(g, k, P) || r || cnt != rows);
            bad += el * EB % 16 || rb * cnt % 16 || so % 16 || cnt < 1;
            bad += (el + (size_t)cnt * g.px) > Q * SS;
            bad += so + cnt * rb > (uint32_t)(k + 1) * rows_region<PREC>() - ROWS_MAXR * 4;
            if (bad) return;
            for (size_t e = 0; e < (size_t)cnt * g.px; ++e) {
              long& q = (load ? src : dst)[so / 2 + e * EB / 2];
              bad += q != -1;
              q = (long)(el + e);
              if (!load) {
                bad += written[el + e] != -1;  // one tile, one copy per element
                written[el + e] = (int)t;
              }
            }
          };
          if (load) face_runs<true>(g, P, k, y0, z, rows, copy);
          else face_runs<false>(g, P, k, y0, z, rows, copy);
          bad += total != rows;
        }
      if (!per[0])
        for (int i = 0; i < rows * 10; ++i) {
          uint32_t off;
          const size_t go = (const char*)row_side<PREC>(g, base, P, i, y0, z, off) - base;
          bad += go % 4 || off % 4 || off + 4 > (uint32_t)rows_stage<PREC>() || go + 4 > Q * SS * EB;
          if (inner) {
            uint32_t o;
            bad += (ptrdiff_t)at0 + (i / 10) * g.px + side_offset<PREC>(g, P, i % 10, o) != (ptrdiff_t)(go / EB);
            bad += o + 4 * (i / 10) != off;
          }
          for (uint32_t h = 0; h < 4 / EB && !bad; ++h) src[(off + h * EB) / 2] = (long)(go / EB + h);
        }
      if (bad) return bad;
      std::vector<int> owner(rows_stage<PREC>() / 2, -1);
      for (int tid = 0; tid < ROWS_CONS; ++tid) {
        const RowPair q = row_pair<PREC>(g, rt.R, rt.tpr, tid);
        for (uint32_t o : {q.xo, q.xo + EB, q.lo, q.yA, q.yB, q.wA, q.wB}) bad += o + EB > (uint32_t)rows_region<PREC>();
        bad += q.xo % (2 * EB);
        const int y = y0 + q.row;
        if (!q.active || y >= ny) continue;
        for (int k = 0; k < 2; ++k) {
          const int x = q.x + k, id = 2 * tid + k;
          if (x >= nx) continue;
          auto is = [&](const std::vector<long>& m, int region, uint32_t off, int arr, int X, int Y, int Z) {
            bad += m[(region * rows_region<PREC>() + off) / 2] != (long)(arr * SS + lin(g, X, Y, Z));
          };
          auto own = [&](int region, uint32_t off) {
            int& o = owner[(region * rows_region<PREC>() + off) / 2];
            bad += o != -1 && o != id;
            o = id;
          };
          const uint32_t xo = q.xo + k * EB;
          is(src, 0, xo, 0, x, y, z);
          is(dst, 0, xo, 0, x, y, z);
          own(0, xo);
          for (int pi = 0; pi < 9; ++pi) {
            const int a = pair_a(pi), d[3] = {cx(a), cy(a), cz(a)}, c[3] = {x, y, z}, n[3] = {nx, ny, nz};
            const int s0 = 1 + 2 * pi, sP = P ? s0 + 1 : s0, sQ = P ? s0 : s0 + 1;
            bool fwd = false, bwd = false;
            int f[3];
            for (int m = 0; m < 3; ++m) {
              f[m] = c[m] + d[m];
              if (per[m]) f[m] = (f[m] + n[m]) % n[m];
              else {
                fwd = fwd || f[m] < 0 || f[m] >= n[m];
                bwd = bwd || c[m] - d[m] < 0 || c[m] - d[m] >= n[m];
              }
            }
            const uint32_t ra = d[0] ? (k ? xo : q.lo) : xo, rbo = d[0] ? (k ? q.yB : q.yA) : xo;
            const uint32_t wo = d[0] ? (k ? q.wB : q.wA) : xo;
            is(src, 1 + 2 * pi, ra, bwd ? sP : sQ, x, y, z);
            is(src, 2 + 2 * pi, rbo, fwd ? sQ : sP, f[0], f[1], f[2]);
            is(dst, 1 + 2 * pi, xo, sQ, x, y, z);
            is(dst, 2 + 2 * pi, wo, sP, f[0], f[1], f[2]);
            own(1 + 2 * pi, xo);
            own(2 + 2 * pi, wo);
            own(1 + 2 * pi, ra);  // nothing is read that another thread overwrites in place
            own(2 + 2 * pi, rbo);
          }
        }
      }
    }
  }
  return bad;
}

int main() {
  std::mt19937 r(3);
  long bad = 0;
  int count = 0;
  for (int nx : {4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 75, 100, 128, 129, 255, 256, 257, 500, 511, 512, 513,
                 560, 567, 568, 576, 577})
    for (int m = 0; m < 8; ++m) {
      const int per[3] = {m & 1, m >> 1 & 1, m >> 2 & 1};
      for (int ny : {2 + (int)(r() % 40), 2 + (int)(r() % 3)}) {
        const int nz = 2 + (int)(r() % 4);
        const long b32 = check<LBM_PREC_F32>(nx, ny, nz, per), b16 = check<LBM_PREC_F16S>(nx, ny, nz, per);
        if (b32 || b16) std::printf("%dx%dx%d periodic %d%d%d: fp32 %ld, 2-byte %ld\n", nx, ny, nz, per[0], per[1], per[2], b32, b16);
        bad += b32 + b16;
        count += 2;
      }
    }
  std::printf("%d grids checked, %ld errors\n", count, bad);
  return bad != 0;
}
