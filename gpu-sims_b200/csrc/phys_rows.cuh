// Row-tile step of the physics mode: persistent blocks that stream whole rows
// through shared memory with bulk copies, so that the collision threads do no
// address arithmetic at all.
//
// A tile is R consecutive rows of one z-plane.  In each of the 19 slot arrays
// its values are one contiguous run of R * px elements, fetched by one
// cp.async.bulk and written back by one (two where a row at a y face comes
// from another place).  Four service warps issue them and resolve everything
// that depends on the row only: the parity, the periodic wraps, and the half-way
// bounce-back of the y and z faces (the same location of the pair's other slot
// array).  The x faces' bounce-back values (one element per row and array) arrive
// by 4-byte cp.async next to the rows.
// Consumer threads own two x-adjacent nodes for the whole launch; every access
// is a fixed offset from a few per-thread bases, the slots at x+1 of the
// c_x = +1 pairs included.
//
// What bounds it.  The row kernels (phys_step_launch.cuh) spend 462 thread
// instructions a node on fp16 storage, half of them addresses, face predicates
// and shuffles, and are bound by their issue; here it is 330, the collision most
// of them, and HBM is the bound of wide grids.  B200, GLUPS (row kernels in
// brackets): fp16 channel 512x128x128 69 = 5.3 TB/s (54), periodic TRT 256^3 76 =
// 5.9 TB/s (57), open duct 512x128x128 67 (51), cavity 160^3 62 (44), 161x97x75
// with Smagorinsky 34.6 (26.2); fp32 channel 41.2 = 6.3 TB/s (39.4), duct 39.1
// (34.9), cavity 160^3 37.1 (33.6), 101^3 38.9 (29.3), 161x97x75 with Smagorinsky
// 30.8 (25.1).
// Four service warps rather than one: each copy is a serial handful of
// instructions, and one warp issuing all 38 of a tile held the block back
// (channel fp16 38.7).  A tile of about 512 nodes keeps the copies long (1 KB
// and up), and five stages of it fit two blocks per SM (2-byte storage).
//
// In place.  Every slot element belongs to one node per launch (phys_kernels.cu),
// so a row of S[1-P] belongs to its own tile and a row of S[P] to the tile of
// the row it is the forward neighbour of; tiles never write each other's rows.
// Elements nobody owns (solid nodes' slots, row padding, x = 0 of the c_x = +1
// pairs beside a wall) are written back as they were read.  Where a face row
// was read from the pair's other array, the elements left unwritten are slots
// whose reader would lie outside the box.
#pragma once
#include "phys_step.cuh"

namespace lbm {
namespace {

constexpr int ROWS_CAP = 576;    // elements of a tile in one slot array
constexpr int ROWS_MAXR = 12;    // rows of a tile
constexpr int ROWS_CONS = 256;   // consumer threads
constexpr int ROWS_SERV = 4;     // service warps, which issue the copies
constexpr int ROWS_MAXST = 5;
// polls of a wait (each try_wait suspends for a while) before the block gives up
// (Ctx::row_wait_polls for the collision's wait for its rows)
constexpr uint32_t ROWS_WAIT_LIMIT = LBM_ROW_WAIT_LIMIT;

// One array's part of a stage: the tile's elements, then a 4-byte slot per
// row for the x face's value.
template <int PREC>
constexpr int rows_region() {
  return ROWS_CAP * (int)sizeof(typename Store<PREC>::T) + ROWS_MAXR * 4;
}
template <int PREC>
constexpr int rows_stage() {
  return Q * rows_region<PREC>();
}
static_assert(rows_region<LBM_PREC_F32>() % 16 == 0 && rows_region<LBM_PREC_F16S>() % 16 == 0,
              "bulk copies start on 16-byte boundaries");

constexpr int ROWS_THREADS = 32 * ROWS_SERV + ROWS_CONS;
// Blocks per SM.  One for Smagorinsky, whose collision spills at 96 registers
// (periodic 256^3 fp32 41.1 GLUPS against 27.1 with two, 128^3 fp16 49.9 against
// 42.8).
template <int PREC, int SGS>
constexpr int rows_blocks() {
  return SGS ? 1 : 2;
}
// Two blocks of 12 warps leave 80 registers a thread at launch (384 * 80 =
// 30,720 a block); the service warpgroup hands its share on:
// 128 * 48 + 256 * 96 = 30,720.
constexpr int ROWS_REGS_SERV = 48, ROWS_REGS_CONS = 96;
static_assert(128 * ROWS_REGS_SERV + ROWS_CONS * ROWS_REGS_CONS <= ROWS_THREADS * 80, "registers of a block");

struct RowTiles {
  int R;            // rows per tile
  int tpr;          // consumer threads per row, two nodes each
  int tiles_y;      // tiles per z-plane
  uint32_t ntiles;
  int stages;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait: false when it ran out or another warp of the block gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t polls) {
  if (mbar_try(bar, parity)) return true;
  for (uint32_t i = 0; i < polls; ++i) {
    if (mbar_try(bar, parity)) return true;
    if (*abort) return false;
  }
  return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}

// A tile of a walk over the grid: first, first + stride, ... in row order.
struct RowWalk {
  int ty, z;      // tile within its plane, plane
  int dty, dz;    // the stride in both
  __host__ __device__ __forceinline__ void start(uint32_t first, uint32_t stride, int tiles_y) {
    z = (int)(first / (uint32_t)tiles_y);
    ty = (int)(first - (uint32_t)z * (uint32_t)tiles_y);
    dz = (int)(stride / (uint32_t)tiles_y);
    dty = (int)(stride - (uint32_t)dz * (uint32_t)tiles_y);
  }
  __host__ __device__ __forceinline__ void next(int tiles_y) {
    ty += dty;
    z += dz;
    if (ty >= tiles_y) {
      ty -= tiles_y;
      ++z;
    }
  }
};

// Row shift of array k's tile rows: (cy, cz) of the pair for Y arrays (even k),
// 0 for X arrays and the rest array.
__host__ __device__ __forceinline__ void array_dir(int k, int& cya, int& czz) {
  // c_y + 1 and c_z + 1 of the nine pairs' forward vectors, two bits each
  constexpr uint32_t CY = [] {
    uint32_t v = 0;
    for (int q = 0; q < 9; ++q) v |= (uint32_t)(cy(pair_a(q)) + 1) << (2 * q);
    return v;
  }();
  constexpr uint32_t CZ = [] {
    uint32_t v = 0;
    for (int q = 0; q < 9; ++q) v |= (uint32_t)(cz(pair_a(q)) + 1) << (2 * q);
    return v;
  }();
  const int q = k > 0 ? (k - 1) >> 1 : 0;
  cya = k > 0 ? (int)((CY >> (2 * q)) & 3u) - 1 : 0;
  czz = k > 0 ? (int)((CZ >> (2 * q)) & 3u) - 1 : 0;
}

// Element offset (from the tile's first element in array 0) of array k's rows
// in a tile away from the y and z faces: where they are loaded from and stored
// to.  X arrays: S[1-P](n); Y arrays: S[P](n + d).
__host__ __device__ __forceinline__ ptrdiff_t array_offset(const PhysGeom& G, int k, int P) {
  if (k == 0) return 0;
  int dy, dz;
  array_dir(k, dy, dz);
  const int s0 = 1 + ((k - 1) & ~1);
  const bool Y = !(k & 1);
  const ptrdiff_t arr = (ptrdiff_t)((Y ? P : 1 - P) + s0) * (ptrdiff_t)G.slot_stride;
  return Y ? arr + (ptrdiff_t)dy * G.px + (ptrdiff_t)dz * (ptrdiff_t)G.pxy : arr;
}

// Array k's rows of any tile: calls copy(element offset from the tile's first
// element in array 0, first row, rows) for every run.  LOAD: where the streamed
// values come from (the pair's other array at a bounce-back face); else where
// the results go.
template <bool LOAD, class F>
__host__ __device__ __forceinline__ void face_runs(const PhysGeom& G, int P, int k, int y0, int z, int rows, F&& copy) {
  const ptrdiff_t SS = (ptrdiff_t)G.slot_stride;
  ptrdiff_t m = array_offset(G, k, P);
  int dy, dz;
  array_dir(k, dy, dz);
  const bool Y = k > 0 && !(k & 1);
  // to the pair's other array: S[P] <-> S[1-P]
  const ptrdiff_t other = k == 0 ? 0 : ((Y ? P : 1 - P) ? -SS : SS);
  // the faces that n + d (Y) or n - d (X) may cross
  const int ey = Y ? dy : -dy, ez = Y ? dz : -dz;
  const bool fy = (ey > 0 && y0 + rows == G.ny) || (ey < 0 && y0 == 0);
  const bool fz = (ez > 0 && z == G.nz - 1) || (ez < 0 && z == 0);
  const ptrdiff_t plain = m;
  if (fz) {
    if (!G.per[2]) m += LOAD ? other : 0;
    else if (Y) m -= (ptrdiff_t)ez * (ptrdiff_t)G.pxy * G.nz;
  }
  const int r = ey > 0 ? rows - 1 : 0;  // the row at the y face
  ptrdiff_t e = m;
  bool own = false;                     // that row comes from (goes) elsewhere
  if (fy) {
    if (!G.per[1]) {
      own = LOAD;
      e = plain + other;
      // a corner link that also wraps in z keeps its wrap
      if (fz && G.per[2] && Y) e -= (ptrdiff_t)ez * (ptrdiff_t)G.pxy * G.nz;
    } else if (Y) {
      own = true;
      e = m - (ptrdiff_t)ey * (ptrdiff_t)G.px * G.ny;
    }
  }
  if (!own) {
    copy(m, 0, rows);
    return;
  }
  copy(e + (ptrdiff_t)r * G.px, r, 1);
  if (rows > 1) {
    const int f = r == 0 ? 1 : 0;
    copy(m + (ptrdiff_t)f * G.px, f, rows - 1);
  }
}

// Entry i of a tile's x-face values (10 per row): its source element's word and
// its place in the stage.  f_a of x = 0 is S[P](0), f_b of x = nx-1 is
// S[1-P](nx) of the forward row.
template <int PREC>
__host__ __device__ __forceinline__ const typename Store<PREC>::T* row_side(const PhysGeom& G, const void* pop, int P,
                                                                            int i, int y0, int z, uint32_t& off) {
  using T = typename Store<PREC>::T;
  const int r = i / 10, e = i - 10 * r, k = e >> 1;
  const int pi = k == 0 ? 0 : k + 2;  // the pairs with c_x = +1: 0, 3, 4, 5, 6
  const int a = pair_a(pi);
  const T* s0 = reinterpret_cast<const T*>(pop) + (size_t)(1 + 2 * pi) * G.slot_stride;
  const T* s1 = s0 + G.slot_stride;
  off = (uint32_t)(1 + 2 * pi + (e & 1)) * rows_region<PREC>() + ROWS_CAP * (uint32_t)sizeof(T) + 4u * (uint32_t)r;
  if (!(e & 1)) return (P ? s1 : s0) + lin(G, 0, y0 + r, z);
  int yn = y0 + r + cy(a), zn = z + cz(a);
  if (G.per[1]) yn = yn < 0 ? yn + G.ny : (yn >= G.ny ? yn - G.ny : yn);
  if (G.per[2]) zn = zn < 0 ? zn + G.nz : (zn >= G.nz ? zn - G.nz : zn);
  return (P ? s0 : s1) + lin(G, sizeof(T) == 2 ? G.nx & ~1 : G.nx, yn, zn);
}

// The same entry of row 0 of a tile away from the y and z faces, from the tile's
// first element in array 0.
template <int PREC>
__host__ __device__ __forceinline__ ptrdiff_t side_offset(const PhysGeom& G, int P, int e, uint32_t& off) {
  const int k = e >> 1, pi = k == 0 ? 0 : k + 2;
  constexpr int EB = sizeof(typename Store<PREC>::T);
  off = (uint32_t)(1 + 2 * pi + (e & 1)) * rows_region<PREC>() + ROWS_CAP * (uint32_t)EB;
  if (!(e & 1)) return (ptrdiff_t)(1 + 2 * pi + P) * (ptrdiff_t)G.slot_stride;
  int dy, dz;
  array_dir(2 + 2 * pi, dy, dz);
  return (ptrdiff_t)(2 + 2 * pi - P) * (ptrdiff_t)G.slot_stride + (ptrdiff_t)dy * G.px +
         (ptrdiff_t)dz * (ptrdiff_t)G.pxy + (EB == 2 ? G.nx & ~1 : G.nx);
}

// The barriers of a block's stages, and its abort mark.
struct RowBars {
  uint32_t full, done;  // shared addresses: rows landed, nodes collided
  uint32_t* loaded;     // shared, per service warp: tiles it has loaded (rows_drain)
  volatile uint32_t* abort;
  unsigned* status;
  __device__ __forceinline__ void give_up() const {
    if ((threadIdx.x & 31) == 0) {
      *abort = 1u;
      atomicOr(status, 4u);
    }
  }
};
// A stage index and its phase parity, in tile order.
struct RowStage {
  uint32_t s = 0, ph = 0;
  __device__ __forceinline__ void next(uint32_t stages) {
    if (++s == stages) {
      s = 0;
      ph ^= 1u;
    }
  }
};

__device__ __forceinline__ bool inner_tile(const PhysGeom& G, int y0, int z, int rows) {
  return y0 > 0 && y0 + rows < G.ny && z > 0 && z < G.nz - 1;
}
// A block that gives up leaves no load in flight.  A tile's `full` phase takes
// the arrivals of all service warps, and they may have stopped at different
// tiles: a warp that loaded `mine` tiles, where the one furthest ahead loaded
// `most`, first arrives for those it left out, and then every load of the block
// shows in the phases of the last `stages` tiles.  Those waits end: a warp loads
// tile t only when tile t - stages is collided, so all have loaded that one, the
// tiles between mine and most lie in different stages, and their phases are the
// stages' current ones.  arrive(stage) makes a warp's whole arrival, wait(stage,
// parity) waits for a phase.
template <class ARRIVE, class WAIT>
__host__ __device__ __forceinline__ void rows_drain(uint32_t mine, uint32_t most, uint32_t stages, ARRIVE&& arrive,
                                                    WAIT&& wait) {
  for (uint32_t t = mine; t < most; ++t) arrive(t % stages);
  for (uint32_t t = most > stages ? most - stages : 0; t < most; ++t) wait(t % stages, (t / stages) & 1u);
}

// The end of a block that gave up (rows_drain), for one service warp.  Out of line:
// inlined, it cost the steps of 2-byte storage with Smagorinsky and a body force
// 3.5 per cent.
__device__ __noinline__ void rows_land(uint32_t full, const volatile uint32_t* counts, uint32_t loaded, uint32_t stages) {
  uint32_t most = 0;
  for (int w = 0; w < ROWS_SERV; ++w) most = max(most, counts[w]);
  rows_drain(
      loaded, most, stages,
      [&](uint32_t s) {
        if ((threadIdx.x & 31) == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], 33;" ::"r"(full + 8 * s) : "memory");
      },
      [&](uint32_t s, uint32_t parity) {
        for (uint32_t i = 0; i < ROWS_WAIT_LIMIT; ++i)
          if (mbar_try(full + 8 * s, parity)) break;
      });
}

constexpr int ROWS_NA = (Q + ROWS_SERV - 1) / ROWS_SERV;  // arrays of a service warp: part, part + ROWS_SERV, ...
constexpr uint64_t ROWS_MOST_BYTES = 1ull << 36;          // of a store (32-bit offsets of 16 bytes, below)

// A block's walk: `count` tiles from tile `first` on, `stride` apart.
struct RowRun {
  RowTiles rt;
  uint32_t first, stride, count;
};

// A service warp's part of a block: loads ahead of the collision and writes back
// behind it.  One lane issues the copies of the warp's arrays: their operands are
// then uniform over the warp, and each costs a handful of instructions.
template <int PREC>
__device__ __forceinline__ void rows_service(const PhysGeom& G, const RowRun& run, void* pop, int P, int part,
                                             uint32_t stage0, const RowBars& B, uint32_t stages, RowStage& st_) {
  using T = typename Store<PREC>::T;
  constexpr uint32_t EB = sizeof(T);
  const int lane = threadIdx.x & 31;
  char* base = reinterpret_cast<char*>(pop);
  const uint32_t row_bytes = (uint32_t)G.px * EB;
  const uint32_t arrays = (uint32_t)((Q + ROWS_SERV - 1 - part) / ROWS_SERV);
  // The warp's arrays away from the y and z faces, in 16-byte units from a
  // tile's first element in array 0 (never negative: an array's rows lie beyond
  // the arrays before it).
  uint32_t off[ROWS_NA];
#pragma unroll
  for (int i = 0; i < ROWS_NA; ++i) {
    off[i] = (uint32_t)((uint64_t)array_offset(G, min(part + ROWS_SERV * i, Q - 1), P) * EB / 16);
    asm volatile("" : "+r"(off[i]));  // not recomputed, nor kept in 64 bits
  }
  // this lane's x-face value of a row: where it lies from the row's first
  // element in array 0 (tiles away from the y and z faces), and its place
  const int side_row = lane < 30 ? lane / 10 : ROWS_MAXR, side_e = lane % 10;
  uint32_t side_dst;
  const ptrdiff_t side_src = side_offset<PREC>(G, P, side_e, side_dst) * (ptrdiff_t)EB;
  RowWalk wl, ws;  // of the loads and of the stores
  wl.start(run.first, run.stride, run.rt.tiles_y);
  ws = wl;
  auto load = [&](uint32_t s) {
    const int z = wl.z, y0 = wl.ty * run.rt.R, rows = min(run.rt.R, G.ny - y0);
    const uint32_t st = stage0 + s * rows_stage<PREC>(), bar = B.full + 8 * s;
    const char* at = base + lin(G, 0, y0, z) * EB;
    const bool in = inner_tile(G, y0, z, rows);
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)rows * row_bytes;
      mbar_arrive_tx(bar, bytes * arrays);
      if (in) {
#pragma unroll
        for (int i = 0; i < ROWS_NA; ++i) {
          const int k = part + ROWS_SERV * i;
          if (k < Q) bulk_load(st + k * rows_region<PREC>(), at + (uint64_t)off[i] * 16, bytes, bar);
        }
      } else {
#pragma unroll 1
        for (int k = part; k < Q; k += ROWS_SERV)
          face_runs<true>(G, P, k, y0, z, rows, [&](ptrdiff_t el, int r, int cnt) {
            bulk_load(st + k * rows_region<PREC>() + (uint32_t)r * row_bytes, at + el * (ptrdiff_t)EB,
                      (uint32_t)cnt * row_bytes, bar);
          });
      }
    }
    __syncwarp();
    if (!G.per[0]) {
      // ten lanes a row, three rows a warp
      for (int r = 3 * part + side_row; r < rows; r += 3 * ROWS_SERV) {
        const char* src = at + side_src + (uint32_t)r * row_bytes;
        uint32_t o = side_dst + 4u * (uint32_t)r;
        if (!in) src = reinterpret_cast<const char*>(row_side<PREC>(G, pop, P, 10 * r + side_e, y0, z, o));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(st + o), "l"(src) : "memory");
      }
    }
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    wl.next(run.rt.tiles_y);
  };
  uint32_t loaded = 0, sl = st_.s;
#pragma unroll 1
  for (; loaded < min(stages, run.count); ++loaded) {
    load(sl);
    if (++sl == stages) sl = 0;
  }
  uint32_t prev = 0;
  bool ok = true;
#pragma unroll 1
  for (uint32_t j = 0; j < run.count; ++j) {
    ok = __all_sync(FULL, mbar_wait(B.done + 8 * st_.s, st_.ph, B.abort, ROWS_WAIT_LIMIT));
    if (!ok) {
      B.give_up();
      break;
    }
    if (lane == 0) {
      const int z = ws.z, y0 = ws.ty * run.rt.R, rows = min(run.rt.R, G.ny - y0);
      const uint32_t st = stage0 + st_.s * rows_stage<PREC>();
      char* at = base + lin(G, 0, y0, z) * EB;
      if (inner_tile(G, y0, z, rows)) {
#pragma unroll
        for (int i = 0; i < ROWS_NA; ++i) {
          const int k = part + ROWS_SERV * i;
          if (k < Q) bulk_store(at + (uint64_t)off[i] * 16, st + k * rows_region<PREC>(), (uint32_t)rows * row_bytes);
        }
      } else {
#pragma unroll 1
        for (int k = part; k < Q; k += ROWS_SERV)
          face_runs<false>(G, P, k, y0, z, rows, [&](ptrdiff_t el, int r, int cnt) {
            bulk_store(at + el * (ptrdiff_t)EB, st + k * rows_region<PREC>() + (uint32_t)r * row_bytes,
                       (uint32_t)cnt * row_bytes);
          });
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      // refill the stage whose stores have left it: the previous tile's, or with
      // two stages this tile's own
      if (stages > 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncwarp();
    ws.next(run.rt.tiles_y);
    if (stages <= 2) prev = st_.s;
    if ((j > 0 || stages <= 2) && loaded < run.count) {
      load(prev);
      ++loaded;
    }
    prev = st_.s;
    st_.next(stages);
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
  if (lane == 0) B.loaded[part] = loaded;
  uint32_t any;  // of the service warps, gave up
  asm volatile("{\n\t.reg .pred P1, P2;\n\tsetp.ne.u32 P1, %1, 0;\n\t"
               "barrier.cta.red.or.pred P2, 1, %2, P1;\n\tselp.b32 %0, 1, 0, P2;\n\t}\n"
               : "=r"(any) : "r"(ok ? 0u : 1u), "n"(32 * ROWS_SERV) : "memory");
  if (any) rows_land(B.full, B.loaded, loaded, stages);
}

// Where a consumer thread's two nodes lie in a stage.
struct RowPair {
  int row, x;              // row within the tile, x of node A
  bool active;             // the thread has a pair
  uint32_t xo;             // byte offset of node A's element (X slots and c_x = 0 Y slots)
  uint32_t lo;             // f_a of node A for the c_x = +1 pairs (x face: the side slot)
  uint32_t yA, yB;         // their f_b of nodes A and B
  uint32_t wA, wB;         // ... and where f*_a of A and B goes
};

template <int PREC>
__host__ __device__ __forceinline__ RowPair row_pair(const PhysGeom& G, int R, int tpr, int tid) {
  constexpr uint32_t EB = sizeof(typename Store<PREC>::T);
  RowPair q;
  q.row = tid / tpr;
  q.active = q.row < R;
  if (!q.active) q.row = 0;
  q.x = q.active ? 2 * (tid - q.row * tpr) : 0;
  const uint32_t r0 = (uint32_t)q.row * (uint32_t)G.px * EB;
  const uint32_t side = ROWS_CAP * EB + 4 * (uint32_t)q.row;
  q.xo = r0 + (uint32_t)q.x * EB;
  q.lo = (!G.per[0] && q.x == 0) ? side : q.xo;
  q.yA = q.wA = q.xo + EB;
  q.yB = q.wB = q.xo + 2 * EB;
  if (q.x == G.nx - 1) {
    if (G.per[0]) q.yA = q.wA = r0;
    else q.yA = side + (EB == 2 && (G.nx & 1) ? 2u : 0u);
    q.yB = q.wB = q.xo + EB;  // node B does not exist
  } else if (q.x + 1 == G.nx - 1) {
    if (G.per[0]) q.yB = q.wB = r0;
    else q.yB = side;  // nx even: the low half of its word
  }
  return q;
}

// One pair of nodes' step on a landed tile: stream from, and collide into, the
// stage at st.
template <int PREC, int COLL, int SGS, bool FORCE, bool WRITE_MOMENTS, bool OPEN>
__device__ __forceinline__ void row_pair_step(const PhysParams& p, const PhysGeom& G,
                                              uint8_t* __restrict__ st, const RowPair& q,
                                              void* __restrict__ pop_v, const uint32_t* __restrict__ links,
                                              float* __restrict__ rho_o, float* __restrict__ u_o,
                                              unsigned* __restrict__ status, int y, int z, uint32_t fl2, int P) {
  using S = Store<PREC>;
  using V2 = Vec2<PREC>;
  using T = typename S::T;
  constexpr int REG = rows_region<PREC>();
  const int x = q.x;
  auto el = [&](int region, uint32_t off) -> T* { return reinterpret_cast<T*>(st + region * REG + off); };
  auto one = [&](int region, uint32_t off) { return S::raw_ld(el(region, off), 0); };
  auto two = [&](int region) {
    const typename V2::V r = V2::ld(el(region, q.xo), 0);
    return make_float2(V2::lo(r), V2::hi(r));
  };
  float2 g[Q];  // .x = node A, .y = node B
  g[0] = two(0);
  static_for<0, 9>([&](auto PI) {
    constexpr int pi = decltype(PI)::value;
    constexpr int a = pair_a(pi), b = pair_b(pi);
    if constexpr (cx(a) == 0) {
      g[a] = two(1 + 2 * pi);
      g[b] = two(2 + 2 * pi);
    } else {
      g[a] = make_float2(one(1 + 2 * pi, q.lo), one(1 + 2 * pi, q.xo + (uint32_t)sizeof(T)));
      g[b] = make_float2(one(2 + 2 * pi, q.yA), one(2 + 2 * pi, q.yB));
    }
  });
  const uint32_t nid = (uint32_t)x + (uint32_t)G.nx * ((uint32_t)y + (uint32_t)G.ny * (uint32_t)z);
  const uint32_t flA = fl2 & 0xffu, flB = fl2 >> 8;
  const bool fluidA = !(flA & FLAG_SOLID), fluidB = !(flB & FLAG_SOLID);
  if (p.any_moving_wall && near_moving(p, x, x + 1 < G.nx ? x + 1 : x, y, z)) {
    auto faces = [&](int xx, auto sel) {
      constexpr bool B = decltype(sel)::value != 0;
      const bool xlo = !G.per[0] && xx == 0, xhi = !G.per[0] && xx == G.nx - 1;
      const bool ylo = !G.per[1] && y == 0, yhi = !G.per[1] && y == G.ny - 1;
      const bool zlo = !G.per[2] && z == 0, zhi = !G.per[2] && z == G.nz - 1;
      static_for<0, 9>([&](auto PI) {
        constexpr int pi = decltype(PI)::value;
        constexpr int a = pair_a(pi), b = pair_b(pi);
        constexpr int DX = cx(a), DY = cy(a), DZ = cz(a);
        const bool fwd = (DX > 0 && xhi) || (DY > 0 && yhi) || (DY < 0 && ylo) || (DZ > 0 && zhi) || (DZ < 0 && zlo);
        const bool bwd = (DX > 0 && xlo) || (DY > 0 && ylo) || (DY < 0 && yhi) || (DZ > 0 && zlo) || (DZ < 0 && zhi);
        float& va = B ? g[a].y : g[a].x;
        float& vb = B ? g[b].y : g[b].x;
        if (bwd) va = fmaf(S::SC, wall_term<a>(p, xx, y, z), va);
        if (fwd) vb = fmaf(S::SC, wall_term<b>(p, xx, y, z), vb);
      });
    };
    faces(x, IC<0>{});
    if (x + 1 < G.nx) faces(x + 1, IC<1>{});
  }
  // links into interior solids: their bounce-back slots are nobody's this
  // launch, so they are read from global memory
  auto solid_fix = [&](int xx, auto sel) {
    constexpr bool B = decltype(sel)::value != 0;
    const T* pop = reinterpret_cast<const T*>(pop_v);
    const uint32_t Lk = links[nid + (B ? 1 : 0)];
    const uint32_t ln = lin32(G, xx, y, z);
    const Wrap w = wrap_terms(G, xx, y, z);
    const bool xlo = !G.per[0] && xx == 0, xhi = !G.per[0] && xx == G.nx - 1;
    const bool ylo = !G.per[1] && y == 0, yhi = !G.per[1] && y == G.ny - 1;
    const bool zlo = !G.per[2] && z == 0, zhi = !G.per[2] && z == G.nz - 1;
    static_for<0, 9>([&](auto PI) {
      constexpr int pi = decltype(PI)::value;
      constexpr int a = pair_a(pi), b = pair_b(pi);
      constexpr int DX = cx(a), DY = cy(a), DZ = cz(a);
      const T* s0 = pop + (size_t)(1 + 2 * pi) * G.slot_stride;
      const T *sP = P ? s0 + G.slot_stride : s0, *sQ = P ? s0 : s0 + G.slot_stride;
      const bool fwd = (DX > 0 && xhi) || (DY > 0 && yhi) || (DY < 0 && ylo) || (DZ > 0 && zhi) || (DZ < 0 && zlo);
      const bool bwd = (DX > 0 && xlo) || (DY > 0 && ylo) || (DY < 0 && yhi) || (DZ > 0 && zlo) || (DZ < 0 && zhi);
      float& va = B ? g[a].y : g[a].x;
      float& vb = B ? g[b].y : g[b].x;
      if (((Lk >> b) & 1u) && !bwd) va = S::raw_ld(sP, ln);
      if (((Lk >> a) & 1u) && !fwd) vb = S::raw_ld(sQ, ln + offs<DX, DY, DZ>(G, w));
    });
  };
  if (fluidA && (flA & FLAG_SOLID_LINK)) solid_fix(x, IC<0>{});
  if (fluidB && (flB & FLAG_SOLID_LINK)) solid_fix(x + 1, IC<1>{});
  // open x faces: the populations entering through them are rebuilt
  if (OPEN && ((flA | flB) & FLAG_OPEN)) {
    if (flA & FLAG_OPEN) {
      auto at = [&](int i) -> float& { return g[i].x; };
      if (x == 0) zou_he<1>(p, S::SC, S::INV, at);
      else zou_he<-1>(p, S::SC, S::INV, at);
    }
    if (flB & FLAG_OPEN) zou_he<-1>(p, S::SC, S::INV, [&](int i) -> float& { return g[i].y; });
  }

  float2 r2, ux2, uy2, uz2;
  collide_t<Ops2, COLL, SGS, FORCE, PREC>(p, CloNet<SGS>{}, g, r2, ux2, uy2, uz2);

  if (WRITE_MOMENTS && q.active && y < G.ny) {
    const uint32_t N = (uint32_t)G.n;
    auto put = [&](float* dst, float a, float b) {
      if (!(G.nx & 1)) {
        *reinterpret_cast<float2*>(dst) = make_float2(a, b);
      } else {  // odd rows start at odd offsets
        dst[0] = a;
        if (x + 1 < G.nx) dst[1] = b;
      }
    };
    put(rho_o + nid, fluidA ? r2.x : 0.f, fluidB ? r2.y : 0.f);
    put(u_o + nid, fluidA ? ux2.x : 0.f, fluidB ? ux2.y : 0.f);
    put(u_o + (size_t)N + nid, fluidA ? uy2.x : 0.f, fluidB ? uy2.y : 0.f);
    put(u_o + 2 * (size_t)N + nid, fluidA ? uz2.x : 0.f, fluidB ? uz2.y : 0.f);
    const bool badA = fluidA && (!(r2.x > 0.f) || !isfinite(r2.x) || !isfinite(ux2.x) || !isfinite(uy2.x) ||
                                 !isfinite(uz2.x));
    const bool badB = fluidB && (!(r2.y > 0.f) || !isfinite(r2.y) || !isfinite(ux2.y) || !isfinite(uy2.y) ||
                                 !isfinite(uz2.y));
    if (badA || badB) atomicOr(status, 1u);
  }

  // Solid nodes' slots hold their neighbours' bounce-back values and stay as
  // they are.  A warp whose pairs are whole (both nodes fluid, or neither) stores
  // pairs; else node by node, in two branches.
  const bool both = fluidA && fluidB, none = !fluidA && !fluidB;
  if (__all_sync(FULL, both || none)) {
    if (both) {
      auto put2 = [&](int region, float a, float b) { V2::st(el(region, q.xo), 0, a, b); };
      put2(0, g[0].x, g[0].y);
      static_for<0, 9>([&](auto PI) {
        constexpr int pi = decltype(PI)::value;
        constexpr int a = pair_a(pi), b = pair_b(pi);
        put2(1 + 2 * pi, g[b].x, g[b].y);  // f*_b -> X
        if constexpr (cx(a) == 0) {
          put2(2 + 2 * pi, g[a].x, g[a].y);  // f*_a -> Y
        } else {
          S::raw_st(el(2 + 2 * pi, q.wA), 0, g[a].x);
          S::raw_st(el(2 + 2 * pi, q.wB), 0, g[a].y);
        }
      });
    }
  } else {
    auto put1 = [&](auto sel) {
      constexpr bool B = decltype(sel)::value != 0;
      auto at = [&](int i) { return B ? g[i].y : g[i].x; };
      S::raw_st(el(0, q.xo), B, at(0));
      static_for<0, 9>([&](auto PI) {
        constexpr int pi = decltype(PI)::value;
        constexpr int a = pair_a(pi), b = pair_b(pi);
        S::raw_st(el(1 + 2 * pi, q.xo), B, at(b));
        if constexpr (cx(a) == 0) S::raw_st(el(2 + 2 * pi, q.xo), B, at(a));
        else S::raw_st(el(2 + 2 * pi, B ? q.wB : q.wA), 0, at(a));
      });
    };
    if (fluidA) put1(IC<0>{});
    if (fluidB) put1(IC<1>{});
  }
}

// Flag bytes of a thread's two nodes; nodes that do not exist read as solid.
__device__ __forceinline__ uint32_t row_flags(const PhysGeom& G, const uint8_t* __restrict__ flags,
                                              const RowPair& q, int y, int z) {
  if (!q.active || y >= G.ny) return 0x0101u;
  const uint32_t nid = (uint32_t)q.x + (uint32_t)G.nx * ((uint32_t)y + (uint32_t)G.ny * (uint32_t)z);
  if (!(G.nx & 1)) return *reinterpret_cast<const uint16_t*>(flags + nid);
  const uint32_t b = q.x + 1 < G.nx ? flags[nid + 1] : (uint32_t)FLAG_SOLID;
  return flags[nid] | b << 8;
}

// A lattice's arrays.
struct RowArrays {
  void* pop;
  const uint8_t* flags;
  const uint32_t* links;
  float *rho, *u;
};

// A consumer thread's part of a block.
template <int PREC, int COLL, int SGS, bool FORCE, bool WRITE_MOMENTS, bool OPEN>
__device__ __forceinline__ void rows_consume(const PhysParams& p, const PhysGeom& G,
                                             const RowRun& run, const RowArrays& D, uint8_t* sm, int tid, int P,
                                             const RowBars& B, uint32_t polls, uint32_t stages, RowStage& st_) {
  const RowPair q = row_pair<PREC>(G, run.rt.R, run.rt.tpr, tid);
  RowWalk w;
  w.start(run.first, run.stride, run.rt.tiles_y);
  int y = w.ty * run.rt.R + q.row, z = w.z;
  uint32_t fl = row_flags(G, D.flags, q, y, z);
  if (polls == 0) {  // testing: no wait at all, not even one that would end at once
    B.give_up();
    return;
  }
  for (uint32_t j = 0; j < run.count; ++j) {
    const int yc = y, zc = z;
    const uint32_t flc = fl;
    if (j + 1 < run.count) {  // the next tile's flags, used one tile later
      w.next(run.rt.tiles_y);
      y = w.ty * run.rt.R + q.row;
      z = w.z;
      fl = row_flags(G, D.flags, q, y, z);
    }
    if (!__all_sync(FULL, mbar_wait(B.full + 8 * st_.s, st_.ph, B.abort, polls))) {
      B.give_up();
      return;
    }
    row_pair_step<PREC, COLL, SGS, FORCE, WRITE_MOMENTS, OPEN>(p, G, sm + st_.s * rows_stage<PREC>(), q,
                                                               D.pop, D.links, D.rho, D.u, B.status, yc, zc, flc, P);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(B.done + 8 * st_.s);
    st_.next(stages);
  }
}

// Set-up of a block: barriers, roles and the share of the registers; cons_warps
// consumer warps take part.  with(f) calls f with the block's work; handed over
// directly instead, 15 of the 32 kernels of a 2-byte format spilled, 428 bytes.
template <int PREC, int COLL, int SGS, bool FORCE, bool WRITE_MOMENTS, bool OPEN, class WITH>
__device__ __forceinline__ void rows_block(uint32_t stages, uint32_t cons_warps, uint32_t polls, unsigned* status, int P,
                                           WITH&& with) {
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ __align__(8) uint64_t bars[2 * ROWS_MAXST];
  __shared__ uint32_t s_abort, s_loaded[ROWS_SERV];
  RowBars B;
  B.full = smem_addr(bars);
  B.done = B.full + 8 * ROWS_MAXST;
  B.loaded = s_loaded;
  B.abort = &s_abort;
  B.status = status;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(B.full + 8 * s, ROWS_SERV * 33);  // the service warps' bytes, and their lanes' cp.async
      mbar_init(B.done + 8 * s, cons_warps);
    }
    s_abort = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int warp = __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0);  // uniform to the compiler
  RowStage st;
  if (warp < ROWS_SERV) {
    if constexpr (rows_blocks<PREC, SGS>() > 1) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ROWS_REGS_SERV));
    with([&](const PhysParams&, const PhysGeom& G, const RowRun& run, const RowArrays& D) {
      rows_service<PREC>(G, run, D.pop, P, warp, smem_addr(sm), B, stages, st);
    });
    if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    return;
  }
  if constexpr (rows_blocks<PREC, SGS>() > 1) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ROWS_REGS_CONS));
  if ((uint32_t)(warp - ROWS_SERV) >= cons_warps) return;
  with([&](const PhysParams& p, const PhysGeom& G, const RowRun& run, const RowArrays& D) {
    rows_consume<PREC, COLL, SGS, FORCE, WRITE_MOMENTS, OPEN>(p, G, run, D, sm, (int)threadIdx.x - 32 * ROWS_SERV, P, B,
                                                              polls, stages, st);
  });
}

// Block b takes tiles b, b + gridDim.x, ...
template <int PREC, int COLL, int SGS, bool FORCE, bool WRITE_MOMENTS, bool OPEN>
__global__ void __launch_bounds__(ROWS_THREADS, rows_blocks<PREC, SGS>())
    k_phys_rows(const __grid_constant__ PhysParams p, RowTiles rt, void* __restrict__ pop_v,
                const uint8_t* __restrict__ flags, const uint32_t* __restrict__ links,
                float* __restrict__ rho_o, float* __restrict__ u_o, unsigned* __restrict__ status, int P,
                uint32_t polls) {
  const RowArrays D{pop_v, flags, links, rho_o, u_o};
  const RowRun run{rt, blockIdx.x, gridDim.x,
                  rt.ntiles <= blockIdx.x ? 0u : (rt.ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x};
  const uint32_t cons_warps = (uint32_t)(rt.R * rt.tpr + 31) / 32;  // warps that have nodes
  rows_block<PREC, COLL, SGS, FORCE, WRITE_MOMENTS, OPEN>((uint32_t)rt.stages, cons_warps, polls, status, P, [&](auto&& f) {
    if (run.count) f(p, p.g, run, D);
  });
}

// Tiles of a grid; R = 0 when a row does not fit (more than 512 nodes, two a
// consumer thread) or its copies would not start on 16-byte boundaries.
inline RowTiles row_tiles(const PhysGeom& G) {
  RowTiles rt{};
  if (G.nx < 4 || G.px % 8 || G.px > ROWS_CAP || (uint64_t)Q * G.slot_stride * 4 >= ROWS_MOST_BYTES) return rt;
  rt.tpr = (G.nx + 1) / 2;
  if (rt.tpr > ROWS_CONS) return rt;
  int R = ROWS_CAP / G.px;
  if (R > ROWS_CONS / rt.tpr) R = ROWS_CONS / rt.tpr;
  if (R > ROWS_MAXR) R = ROWS_MAXR;
  if (R > G.ny) R = G.ny;
  rt.tiles_y = (G.ny + R - 1) / R;
  rt.R = (G.ny + rt.tiles_y - 1) / rt.tiles_y;  // as even as the count allows
  rt.ntiles = (uint32_t)rt.tiles_y * (uint32_t)G.nz;
  rt.stages = ROWS_MAXST;
  return rt;
}

// fp32 stages (45 KB) leave room for one block of five an SM or two of two.
// Deep prefetch wins where the store streams from HBM (channel 512x128x128 41.6
// against 38.6 GLUPS, cavity 160^3 37.6 against 34.4); where it stays in the
// 126 MB L2, twice the consumer warps do (101^3 38.8 against 31.2, 96^3 38.2
// against 29.8).  With Smagorinsky there is one block an SM in any case
// (rows_blocks).
constexpr size_t ROWS_DEEP_BYTES = 120000000;
inline bool rows_deep(const PhysGeom& G, int precision, bool smag) {
  return precision == LBM_PREC_F32 && (smag || 76 * G.slot_stride > ROWS_DEEP_BYTES);
}
// Persistent blocks of the chip's 148 SMs.
inline uint32_t rows_chip_blocks(const PhysGeom& G, int precision, bool smag) {
  return smag || rows_deep(G, precision, smag) ? 148 : 296;
}

// Where row tiles are the default: where they beat the row kernels
// (phys_step_launch.cuh), measured on B200 over 56 row lengths from 66 to 512,
// three sections and 26 thin boxes, both collisions, with and without
// Smagorinsky, in graphs and in single steps (1,592 timings).  Ratios of the
// two times, row tiles' to row kernels':
//  * `used`, the share of the node slots of all blocks' rounds that hold nodes
//    (tiles not filled by whole rows, a plane's ragged last tile, a last round of
//    few blocks), decides most: odd rows in fp32 0.64-0.97 from 62 per cent on; with
//    Smagorinsky, one block an SM, fp16 257 x 97 x 120 (50) 1.31, 181 x 97 x 120 (70)
//    1.10, 97 x 140 x 140 (93) 0.81;
//  * what it replaces: the pair kernels are at their best where rows fill their
//    64-wide warps (`whole`), fp32 384 x 140 x 140 1.11, 512 x 140 x 140 0.95, fp16 with
//    Smagorinsky 448 x 140 x 140 1.09, 112 x 140 x 140 0.87, 512 x 97 x 120 0.90; so is
//    the one-node kernel, which odd rows with Smagorinsky take, at 32: 95 x 97 x 120
//    1.12, 97 x 97 x 120 0.90;
//  * tiles at a y face take twice the copies: one to three a plane 1.0-1.9, four
//    of one row each 1.0-1.3, five of several rows 0.6-0.8; two planes of z 1.0-1.5;
//  * few tiles: fp32 127 x 64 x 64 (1,024) 1.09, 67 x 300 x 24 (1,032) 0.76, fp16 75 x 64 x 64
//    (704, 68 per cent used) 1.20, 71^3 (781, 79) 0.76, whole rows 256 x 256 x 8 (1,024) 1.15;
//  * rows below 66 nodes waste padding and tiles: 64^3 fp16 22.8 against 30.2 GLUPS.
// Open x faces cost the row kernels a launch of their own: 128^3 fp16 with
// Smagorinsky 0.82, without the faces 1.03.
// A body force where the one-node kernel would run (odd rows, even ones that are no
// pairs', open faces) has lines of its own (`fill` and the number of tiles), which
// time alone does not draw: that kernel rounds j / rho and the half force apart, the
// packed collision here in one multiply-add, and 2-byte stores carry that into
// results 2e-3 apart after 50 steps, so a line moved is a result changed.  On both
// sides of them a time is lost: bf16 77 x 63 x 81 TRT 0.87, fp32 with Smagorinsky 437
// x 97 x 46 0.90 and 201 x 48 x 75 1.13, fp16 with Smagorinsky 257 x 80 x 101 1.24 of
// the row kernels' time.
// Inside the other lines 1 in 50 of the timings is slower by more than 4 per cent,
// the worst by 10 (81 x 97 x 120, periodic, TRT, Smagorinsky, fp32, single steps).
inline bool row_tiles_pay(const PhysParams& p, const lbm_desc& d) {
  const PhysGeom& G = p.g;
  const bool f32 = d.precision == LBM_PREC_F32, smag = p.smag_cs > 0.f, odd = G.nx % 2 != 0;
  const RowTiles rt = row_tiles(G);
  if (rt.R == 0 || G.nx < 66) return false;
  const int wide = (G.nx + 63) / 64 * 64;
  const bool whole = !odd && 20 * wide <= 23 * G.nx;
  const int fill = 100 * rt.R * G.nx / 512;  // per cent of a tile
  if (f32 ? fill < 74 : !odd && fill < 76) return false;
  const uint32_t nt = rt.ntiles, blocks = rows_chip_blocks(G, d.precision, smag);
  const bool force = p.accel[0] != 0.f || p.accel[1] != 0.f || p.accel[2] != 0.f;
  if (force && (!step_pairs(G.nx) || p.any_open)) return nt >= (whole ? (f32 ? 12000u : 4000u) : (f32 ? 1000u : 700u));
  // per mille
  const int used = (int)(1000 * (uint64_t)G.n / (512ull * blocks * ((nt + blocks - 1) / blocks)));
  if (rt.tiles_y < (whole ? 12 : smag || rt.R < 5 ? 5 : 3)) return false;
  if (G.nz < (smag && !odd ? 5 : 4) && !(odd && !f32 && !smag && used >= 750)) return false;
  if (p.any_open) return nt >= (whole ? (f32 ? 12000u : 4000u) : (f32 ? 1000u : 700u));
  if (whole)
    return nt >= (f32 ? 12000u : 4000u) && used * wide >= G.nx * (f32 ? (smag ? 800 : 900) : (smag ? 920 : 720));
  if (!smag) return nt >= (f32 ? 1030u : 700u) && used >= (f32 ? 620 : nt >= 1000 ? 450 : G.per[0] ? 660 : 750);
  if (!odd) return nt >= (rt.R < 5 ? 1500u : 1030u) && used >= 700;
  const bool many = nt >= (f32 ? 5000u : 2400u);
  return nt >= 800 && used >= (many ? 720 : 800) &&
         used * ((G.nx + 31) / 32 * 32) >= G.nx * (!many ? 880 : d.collision == LBM_COLL_TRT ? 870 : 800);
}

template <int PREC, int COLL, int SGS, bool FORCE, bool WM, bool OPEN>
cudaError_t launch_row_tiles(const Ctx& c, int P, cudaStream_t s) {
  RowTiles rt = row_tiles(c.pp.g);
  if (PREC == LBM_PREC_F32 && !rows_deep(c.pp.g, PREC, SGS)) rt.stages = 2;
  const size_t smem = (size_t)rt.stages * rows_stage<PREC>();
  auto* fn = &k_phys_rows<PREC, COLL, SGS, FORCE, WM, OPEN>;
  // The limit belongs to the kernel, which all lattices of the process share (other
  // threads' and captured graphs' among them): always that of the most stages,
  // never lowered to this launch's.
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ROWS_MAXST * rows_stage<PREC>());
  if (e != cudaSuccess) return e;
  const uint32_t most = c.row_blocks ? (uint32_t)c.row_blocks : rows_chip_blocks(c.pp.g, PREC, SGS);
  const dim3 grd(rt.ntiles < most ? rt.ntiles : most);
  fn<<<grd, ROWS_THREADS, smem, s>>>(c.pp, rt, c.pop, c.flags, c.links, c.rho, c.u, c.status, P, c.row_wait_polls);
  return cudaGetLastError();
}

template <int PREC, int COLL, int SGS, bool FORCE>
cudaError_t rows_wm(const Ctx& c, int P, bool wm, cudaStream_t s) {
  if (c.pp.any_open)
    return wm ? launch_row_tiles<PREC, COLL, SGS, FORCE, true, true>(c, P, s)
              : launch_row_tiles<PREC, COLL, SGS, FORCE, false, true>(c, P, s);
  return wm ? launch_row_tiles<PREC, COLL, SGS, FORCE, true, false>(c, P, s)
            : launch_row_tiles<PREC, COLL, SGS, FORCE, false, false>(c, P, s);
}
template <int PREC, int COLL>
cudaError_t rows_coll(const Ctx& c, int P, bool wm, cudaStream_t s) {
  const bool force = c.pp.accel[0] != 0.f || c.pp.accel[1] != 0.f || c.pp.accel[2] != 0.f;
  if (c.pp.smag_cs > 0.f)
    return force ? rows_wm<PREC, COLL, 1, true>(c, P, wm, s) : rows_wm<PREC, COLL, 1, false>(c, P, wm, s);
  return force ? rows_wm<PREC, COLL, 0, true>(c, P, wm, s) : rows_wm<PREC, COLL, 0, false>(c, P, wm, s);
}

}  // namespace
}  // namespace lbm

#define LBM_DEFINE_PHYS_ROWS(NAME, PREC)                                            \
  namespace lbm {                                                                   \
  cudaError_t NAME(const Ctx& c, int parity, bool write_moments, cudaStream_t s) {  \
    return c.d.collision == LBM_COLL_TRT                                            \
               ? rows_coll<PREC, LBM_COLL_TRT>(c, parity, write_moments, s)         \
               : rows_coll<PREC, LBM_COLL_BGK>(c, parity, write_moments, s);        \
  }                                                                                 \
  }
