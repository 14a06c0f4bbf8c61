// fdtd_tma.cuh - the field sub-cycle of the resident simulation (fdtd_ratio 1):
// one block per patch, the patch staged by TMA, the sub-cycle in registers.
//
// One launch advances the fields by one particle step: H(dt/4), E(dt/2),
// H(dt/2), E(dt/2), H(dt/4) (EM3_1.cu:2-17 and EM3.cu:2-43, called as the
// sub-cycle of electricmagneticfield6.m:146-151), with the same arithmetic as
// the general kernel of fdtd.cuh.
//
// Work: the grid (n_r + 1 columns x n_z + 1 rows of Yee points) is cut into
// tiles of 26 columns x (R - 6) rows.  A block owns a patch of 32 columns x R
// rows around its tile (3 halo columns and rows on each side: the five
// sub-updates need two on the low side and three on the high side, and one
// more on the low side lets it assemble every gather quad of its tile
// from values it computed).  Each of its warps holds a segment of S
// consecutive rows in registers - lane l column l: Er, Ez, H and the two
// current terms - so vertical neighbours are registers and horizontal ones
// shuffles; between segments one row of Er or H goes through shared memory per
// update.  The halo is recomputed by each block instead of exchanged: 1.35 times
// the points at R = 64.  (A warp per patch of 32 x 12 recomputed 2.5 times the
// points: 1024 x 4096 cells in 59 us, 31M warp instructions.)
//
// Staging: one thread of each block issues five 2D tensor copies (Er, Ez, H as
// stored, Jr, Jz as 64-bit fixed point) of its patch into the block's staging
// area, completing on its mbarrier.  Once the registers hold the patch the area
// is free, and the copies of the block's next patch go out before the current
// one is computed.  Blocks walk the work items grid-stride.  The tiles are
// written to a second set of fields: a patch
// staged after its neighbours' tiles were written still reads the old fields
// in its halo.
//
// TMA copies want 16-byte aligned starting columns: each box starts at the
// patch's first column rounded down to a 16-byte boundary and is wide enough
// (36 floats, 34 doubles or 64-bit counters) to cover the 32 patch columns
// from there; a lane reads its column at that offset.  Points outside the
// grid (negative or beyond the extent) arrive as zeros and are never updated.
//
// Every wait on an mbarrier is bounded; a block whose copy has not completed
// after the bound sets the cell's *err, waits (bounded) once more for that
// copy and returns.
#pragma once
#include <cuda.h>
#include "fdtd.cuh"

namespace gasatt {

constexpr int kTmaTileW = 26;                 // output columns per tile
constexpr int kTmaPatchW = 32;                // patch columns (one per lane)
constexpr int kTmaHalo = 3;                   // halo columns / rows on each side
constexpr unsigned kTmaWaitLimit = 1u << 22;  // try_wait rounds before giving up

// The patch of knob value K (fdtd_tile_rows): W warps of S rows each, and how
// many blocks an SM is to hold.  (32 warps of 64 registers for 12 and 16, which spill
// 12 to 16 bytes a thread, and 68 in the FP32 batch; 20 spills none.)
template <int K> struct TmaShape;
template <> struct TmaShape<12> { static constexpr int W = 4, S = 4; };
template <> struct TmaShape<16> { static constexpr int W = 8, S = 4; };
template <> struct TmaShape<20> { static constexpr int W = 8, S = 8; };
__host__ __device__ constexpr int tma_warps(int k) { return k == 12 ? 4 : 8; }
__host__ __device__ constexpr int tma_rows(int k) { return k == 12 ? 16 : k == 16 ? 32 : 64; }
__host__ __device__ constexpr int tma_blocks(int k) { return k == 12 ? 8 : k == 16 ? 4 : 2; }
__host__ __device__ constexpr bool tma_rows_ok(int k) { return k == 12 || k == 16 || k == 20; }

// tiles of a grid of n_r x n_z cells
inline int tma_tiles_x(int nr) { return (nr + kTmaTileW) / kTmaTileW; }
inline int tma_tiles(int k, int nr, int nz) {
  const int h = tma_rows(k) - 2 * kTmaHalo;
  return tma_tiles_x(nr) * ((nz + h) / h);
}

// staging box widths (elements): 32 columns from an aligned start below the
// patch's first column
template <typename T> struct TmaBox { static constexpr int w = sizeof(T) == 4 ? 36 : 34; };

// ------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\t"
               "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// true once the phase with the given parity has completed; false after the bound
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (unsigned it = 0; it < kTmaWaitLimit; ++it) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    if (done) return true;
  }
  return false;
}
// 2D tiled tensor copy global -> shared (no multicast), completion on bar
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// ------------------------------------------------------------ layout
// A block's staging area for R patch rows (Er, Ez, H in T, Jr, Jz in 64 bits;
// each 128-byte aligned), then its mbarrier.
template <typename T, int R>
struct TmaStage {
  static constexpr size_t up(size_t b) { return (b + 127) & ~(size_t)127; }
  static constexpr size_t field_bytes = up((size_t)TmaBox<T>::w * R * sizeof(T));
  static constexpr size_t cur_bytes = up((size_t)34 * R * 8);
  static constexpr size_t bytes = 3 * field_bytes + 2 * cur_bytes;
  static constexpr size_t block_bytes = bytes + 128;
  // bytes one patch's five copies deliver (whole boxes, out-of-bounds fill included)
  static constexpr uint32_t tx_bytes =
      (uint32_t)(3 * (size_t)TmaBox<T>::w * R * sizeof(T) + 2 * (size_t)34 * R * 8);
};

struct TmaMaps {
  CUtensorMap er, ez, h, jr, jz;
};

// One gas cell's field update as the kernel sees it: its tensor maps (the
// field and current buffers read in this step), where the tile is written
// (the other field buffer in T, the other current buffer cleared, FP32 gather
// quads),
// the coefficients and its tile grid.  A single cell passes it as a kernel
// parameter; a batch keeps one per cell in global memory.
struct FdtdInst {
  TmaMaps maps;
  void *Er, *Ez, *H;
  unsigned long long *Jr_next, *Jz_next;
  // per column i in [0, n_r]: {1/V scaled from fixed point, coefficient of
  // H(i) and of H(i-1) in the Ez update} (FdtdColumn), precomputed on the host
  // with the expressions the kernels of fdtd.cuh evaluate per thread
  const double *colc;
  ExtraCurrent xj;
  FieldQuads q;
  FdtdCoef c;
  double chr4, chz4, chr2, chz2;   // H update factors h/(mu dr), h/(mu dz) for h = dt/4, dt/2
  int nr, nz, ldf, ldj;
  unsigned flags;
  int tiles_x, ntiles;
  unsigned *err;              // set when a tile copy of this cell did not complete
};

// Work of a launch: tile t of one cell, or entry t of a table of (cell, tile)
// pairs over the cells of a batch.
struct FdtdWork {
  const FdtdInst *inst;       // one cell, or the batch's cells
  const int2 *table;          // null for one cell; else (cell, tile) per work item
  int ntiles;                 // work items
  __device__ __forceinline__ const FdtdInst &at(int t, int &lt) const {
    if (!table) { lt = t; return *inst; }
    const int2 e = table[t];
    lt = e.y;
    return inst[e.x];
  }
};

// tile t of a tiles_x-wide row-major tile grid -> the patch origin (x0, y0)
__device__ __forceinline__ void tma_patch_origin(int t, int tiles_x, int rows, int &x0, int &y0) {
  const int ty = t / tiles_x, tx = t - ty * tiles_x;
  x0 = tx * kTmaTileW - kTmaHalo;
  y0 = ty * (rows - 2 * kTmaHalo) - kTmaHalo;
}

// issue the copies of work item t into the staging area (one thread)
template <typename T, int R>
__device__ __forceinline__ void tma_issue_item(const FdtdWork &W, int t, unsigned char *stage,
                                               uint64_t *bar) {
  using S = TmaStage<T, R>;
  constexpr int al = 16 / (int)sizeof(T);
  int lt, x0, y0;
  const FdtdInst &I = W.at(t, lt);
  tma_patch_origin(lt, I.tiles_x, R, x0, y0);
  const int xf = x0 & ~(al - 1), xj = x0 & ~1;       // floor to a 16-byte column
  const TmaMaps &M = I.maps;
  mbar_expect_tx(bar, S::tx_bytes);
  tma_load_2d(stage, &M.er, xf, y0, bar);
  tma_load_2d(stage + S::field_bytes, &M.ez, xf, y0, bar);
  tma_load_2d(stage + 2 * S::field_bytes, &M.h, xf, y0, bar);
  tma_load_2d(stage + 3 * S::field_bytes, &M.jr, xj, y0, bar);
  tma_load_2d(stage + 3 * S::field_bytes + S::cur_bytes, &M.jz, xj, y0, bar);
}

// The sub-cycle on the work items of W (cells on the padded layout: row
// strides ldf for the fields, ldj for the currents), patches of shape K.
// The field arithmetic is that of fdtd_tiled (fdtd.cuh); the per-column
// coefficients come from the cell's table, the current terms of the two E
// updates are formed once per patch.
template <typename T, int K>
__device__ __forceinline__ void fdtd_block_body(const FdtdWork &W) {
  constexpr int NW = TmaShape<K>::W, S = TmaShape<K>::S, R = NW * S;
  using St = TmaStage<T, R>;
  static_assert(R == tma_rows(K) && NW == tma_warps(K) && S > kTmaHalo, "patch shape");
  constexpr int BW = TmaBox<T>::w, al = 16 / (int)sizeof(T);
  constexpr unsigned FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(128) unsigned char smem[];
  // the rows of a segment that its neighbours read: first and last Er (in two
  // buffers by turns: an E update reads one while others write the other),
  // last H and Ez
  __shared__ double s_first[2][NW][32], s_last[2][NW][32], s_h[NW][32], s_ez[NW][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + St::bytes);
  const int ntiles = W.ntiles, stride = gridDim.x;
  int t = blockIdx.x;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0 && t < ntiles) tma_issue_item<T, R>(W, t, smem, bar);
  for (int k = 0; t < ntiles; t += stride, ++k) {
    int lt, x0, y0;
    const FdtdInst &I = W.at(t, lt);
    tma_patch_origin(lt, I.tiles_x, R, x0, y0);
    y0 += w * S;                           // the segment's first row
    const int nr = I.nr, nz = I.nz;
    const unsigned flags = I.flags;
    const bool endcopy = (flags & GASATT_Q_ER_END_COPY) != 0;
    const bool jsign = (flags & GASATT_Q_EZ_AXIS_JSIGN) != 0;
    const double dt_eps = I.c.dt_eps, dt_eps_dz = I.c.dt_eps_dz, axis = I.c.axis;
    const int col = x0 + lane;
    const int of = x0 - (x0 & ~(al - 1)), oj = x0 - (x0 & ~1);
    const bool colH = col >= 0 && col < nr;
    // Every point of the patch is updated by the same expression: no in-grid
    // update reads a point outside the grid (the boundary rules never reach
    // past the edge), so the values those points take do not matter.  The
    // rules that keep an in-grid point from the interior expression become
    // coefficients: Ez on the axis (col 0) takes (+J term, axis factor, 0),
    // Ez at col n_r and beyond is left as it is (0, 0, 0); Er rows 0 and n_z
    // are fixed up after each E update.  (Read while the copies are in flight.)
    double iv = 0.0, ezp = 0.0, ezm = 0.0;
    if (colH) {
      iv = I.colc[3 * col];
      ezp = col == 0 ? axis : I.colc[3 * col + 1];
      ezm = I.colc[3 * col + 2];            // 0 on the axis
    }
    const bool ok = __syncthreads_and(mbar_wait(bar, (uint32_t)(k & 1)));
    if (!ok) {
      if (threadIdx.x == 0) {
        atomicOr(I.err, 1u);
        mbar_wait(bar, (uint32_t)(k & 1));          // the copy still owns the area
      }
      break;
    }
    // the column's segment: fields, and the current terms of the E updates
    // (jr: dt/eps (J_r(j-1) + J_r(j)) / 2; jz: the same over columns i-1, i,
    // or on the axis minus the signed dt/eps J_z term)
    double er[S], ez[S], h[S], jr[S], jz[S];
    {
      const T *gEr = reinterpret_cast<const T *>(smem);
      const T *gEz = reinterpret_cast<const T *>(smem + St::field_bytes);
      const T *gH = reinterpret_cast<const T *>(smem + 2 * St::field_bytes);
      const long long *gJr = reinterpret_cast<const long long *>(smem + 3 * St::field_bytes);
      const long long *gJz = reinterpret_cast<const long long *>(smem + 3 * St::field_bytes + St::cur_bytes);
      const ExtraCurrent xj = I.xj;
      // row r of the segment (r = -1: the row below it)
      auto current = [&](const long long *g, const unsigned long long *x, int r) {
        double a = (double)g[lane + oj + (w * S + r) * 34];
        if (x) {
          const int row = y0 + r;
          if (colH && row >= 0 && row < nz) a = a + (double)(long long)x[col + (int64_t)row * I.ldj] * xj.rel;
        }
        return a * iv;
      };
      double below = w > 0 ? current(gJr, xj.Jr, -1) : 0.0;
#pragma unroll
      for (int r = 0; r < S; ++r) {
        const int sf = lane + of + (w * S + r) * BW;
        er[r] = (double)gEr[sf];
        ez[r] = (double)gEz[sf];
        h[r] = (double)gH[sf];
        const double a = current(gJr, xj.Jr, r);
        jr[r] = dt_eps * (below + a) / 2;
        below = a;
        jz[r] = current(gJz, xj.Jz, r);
      }
    }
    __syncthreads();
    // the area is free: the block's next patch is fetched while this one is computed
    if (threadIdx.x == 0 && t + stride < ntiles) {
      fence_proxy_async_smem();
      tma_issue_item<T, R>(W, t + stride, smem, bar);
    }
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const double left = __shfl_up_sync(FULL, jz[r], 1);
      const double jt = jsign ? dt_eps * jz[r] : -(dt_eps * jz[r]);
      jz[r] = col == 0 ? -jt : (colH ? dt_eps * (left + jz[r]) / 2 : 0.0);
    }
    // segment rows of grid rows 0 and n_z (Er there: zero, or the end copies)
    const int r0 = -y0, rn = nz - y0;
    const bool edge_rows = (r0 >= 0 && r0 < S) || (rn >= 0 && rn < S);
    // the segments above and below (the patch's first and last read their own
    // row instead: halo points, whose values do not matter)
    const int up = w + 1 < NW ? w + 1 : w, dn = w > 0 ? w - 1 : 0;
    auto publish_e = [&](int b) {
      s_first[b][w][lane] = er[0];
      s_last[b][w][lane] = er[S - 1];
      __syncthreads();
    };
    auto h_update = [&](double chr, double chz, int b) {
      const double above = s_first[b][up][lane];
#pragma unroll
      for (int r = 0; r < S; ++r) {
        const double ezr = __shfl_down_sync(FULL, ez[r], 1);
        const double e1 = r + 1 < S ? er[r + 1 < S ? r + 1 : r] : above;
        h[r] = h[r] + (chr * (ezr - ez[r]) - chz * (e1 - er[r]));
      }
    };
    auto e_update = [&](int b) {
      s_h[w][lane] = h[S - 1];
      __syncthreads();
      const double hb = s_h[dn][lane];
      double ne[S];
#pragma unroll
      for (int r = 0; r < S; ++r) {
        const double hl = __shfl_up_sync(FULL, h[r], 1);
        ne[r] = er[r] - jr[r] - dt_eps_dz * (h[r] - (r > 0 ? h[r > 0 ? r - 1 : 0] : hb));
        ez[r] = ez[r] - jz[r] + ezp * h[r] + ezm * hl;
      }
      if (edge_rows) {
        const double eu = s_first[b][up][lane], ed = s_last[b][dn][lane];
#pragma unroll
        for (int r = 0; r < S; ++r) {
          if (r == r0) ne[r] = endcopy ? (r + 1 < S ? er[r + 1 < S ? r + 1 : r] : eu) : 0.0;
          if (r == rn) ne[r] = endcopy ? (r > 0 ? er[r > 0 ? r - 1 : 0] : ed) : 0.0;
        }
      }
#pragma unroll
      for (int r = 0; r < S; ++r) er[r] = ne[r];
    };
    publish_e(0);
    h_update(I.chr4, I.chz4, 0);
    e_update(0);
    publish_e(1);
    h_update(I.chr2, I.chz2, 1);
    e_update(1);
    publish_e(0);
    h_update(I.chr4, I.chz4, 0);
    // write back the tile: columns [3, 29) and rows [3, R - 3) of the patch
    T *Er = reinterpret_cast<T *>(I.Er), *Ez = reinterpret_cast<T *>(I.Ez), *H = reinterpret_cast<T *>(I.H);
    unsigned long long *Jr_next = I.Jr_next, *Jz_next = I.Jz_next;
    const int ldf = I.ldf, ldj = I.ldj;
    const bool out_col = lane >= kTmaHalo && lane < kTmaHalo + kTmaTileW && col <= nr;
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const int row = y0 + r, pr = w * S + r;
      if (pr < kTmaHalo || pr >= R - kTmaHalo || row > nz) continue;
      if (!out_col) continue;
      if (col < nr) Er[col + (int64_t)row * ldf] = (T)er[r];
      if (row < nz) Ez[col + (int64_t)row * ldf] = (T)ez[r];
      if (col < nr && row < nz) {
        H[col + (int64_t)row * ldf] = (T)h[r];
        const int64_t g = col + (int64_t)row * ldj;
        Jr_next[g] = 0;
        Jz_next[g] = 0;
      }
    }
    if (sizeof(T) == 4 && I.q.er) {
      // FP32 form: whole gather quads from the fields rounded to float, corner
      // columns from the lane below by shuffle, corner rows from the segments
      // above and below
      const FieldQuads q = I.q;
      s_h[w][lane] = h[S - 1];
      s_ez[w][lane] = ez[S - 1];
      __syncthreads();
      const float e_up = (float)s_first[0][up][lane], z_dn = (float)s_ez[dn][lane], h_dn = (float)s_h[dn][lane];
      float fe[S + 1], fz[S + 1], fh[S + 1];     // fe[r]: row r; fz[r], fh[r]: row r - 1
      fe[S] = e_up; fz[0] = z_dn; fh[0] = h_dn;
#pragma unroll
      for (int r = 0; r < S; ++r) {
        fe[r] = (float)er[r];
        fz[r + 1] = (float)ez[r];
        fh[r + 1] = (float)h[r];
      }
      const bool lo0 = col > 0, hi0 = col > nr - 1;   // corner column c0 = col - 1, c1 = col - 1
#pragma unroll
      for (int r = 0; r < S; ++r) {
        const int row = y0 + r, pr = w * S + r;
        if (pr < kTmaHalo || pr >= R - kTmaHalo || row > nz) continue;     // (the same for the whole warp)
        const float eu0 = __shfl_up_sync(FULL, fe[r], 1), eu1 = __shfl_up_sync(FULL, fe[r + 1], 1);
        const float zd0 = __shfl_down_sync(FULL, fz[r], 1), zd1 = __shfl_down_sync(FULL, fz[r + 1], 1);
        const float hu0 = __shfl_up_sync(FULL, fh[r], 1), hu1 = __shfl_up_sync(FULL, fh[r + 1], 1);
        if (!out_col) continue;
        const bool ra_lo = row > 0, rb_lo = row > nz - 1;   // quad rows ra = row - 1, rb = row - 1
        if (row < nz)
          q.er[col + (int64_t)row * (nr + 1)] =
              make_float4(lo0 ? eu0 : fe[r], hi0 ? eu0 : fe[r], lo0 ? eu1 : fe[r + 1], hi0 ? eu1 : fe[r + 1]);
        if (col < nr)
          q.ez[col + (int64_t)row * nr] =
              make_float4(ra_lo ? fz[r] : fz[r + 1], ra_lo ? zd0 : zd1, rb_lo ? fz[r] : fz[r + 1],
                          rb_lo ? zd0 : zd1);
        const float ha0 = ra_lo ? hu0 : hu1, ha = ra_lo ? fh[r] : fh[r + 1];
        const float hb0 = rb_lo ? hu0 : hu1, hb = rb_lo ? fh[r] : fh[r + 1];
        q.h[col + (int64_t)row * (nr + 1)] =
            make_float4(lo0 ? ha0 : ha, hi0 ? ha0 : ha, lo0 ? hb0 : hb, hi0 ? hb0 : hb);
      }
    }
  }
}

// the per-column table of FdtdInst::colc for n_r columns: {1/V scaled, Ez
// coefficients of H(i) and H(i-1)} (the expressions fdtd_tiled evaluates)
inline void fdtd_column_table(int nr, const FdtdCoef &c, const double *invV, unsigned flags,
                              double *out) {
  const double inv_dr = 1 / c.dr;
  for (int i = 0; i < nr; ++i) {
    const double ri = ((flags & GASATT_Q_EZ_RSHIFT) ? (i + 1) : i) * c.dr;
    out[3 * i] = invV[i];
    out[3 * i + 1] = i > 0 ? c.dt_eps * (1 / (2 * ri) + inv_dr) : 0.0;
    out[3 * i + 2] = i > 0 ? c.dt_eps * (1 / (2 * ri) - inv_dr) : 0.0;
  }
}

}  // namespace gasatt
