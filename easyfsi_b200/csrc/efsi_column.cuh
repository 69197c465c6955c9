// Column-marching stencil kernels of the pressure solver's finest level: the
// V-cycle's sweeps and restriction and the CG direction + SpMV, for levels
// wide enough along k (nz >= 40, in efsi_fv_plan_create).
//
// A block of 32 x 4 threads owns a 64 (k) x 8 (j) column tile and a chunk of
// planes [ib, ie) along i.  A thread owns 2 x 2 cells of every plane: k and
// k + 1, j and j + 1, both even.  It marches with its cells' values of planes
// i - 1, i and i + 1 in registers, so that of a plane's stencil inputs only
// the new plane's centres and the cells around the 2 x 2 patch are read from
// shared memory, two doubles a load: 12 shared loads per four cells where the
// one-cell-per-thread march (efsi_march.cuh) takes 36.  One elected thread
// streams the planes (value tiles with a one-cell halo, right-hand side and
// other plain tiles, the stencil mask) into a ring of stages with TMA
// (cp.async.bulk.tensor, no multicast), one mbarrier per stage.
//
// Cells whose stencil is whole -- fluid, every face open or on the domain's
// boundary -- take a path without per-face selection: the axis tables hold
// zero coefficients at the boundary, so the closed faces there add exact
// zeros, as the selected form does.  A warp with any other cell (next to an
// obstacle) takes the selected form for all of its cells, and levels with
// Dirichlet weights or an interface diagonal (kAux) always do.
//
// The 2 x 2 x 2 children of a coarse cell belong to one thread: the
// prolongation needs one coarse value for its cells and four for the patch's
// neighbours per plane pair, added in registers, and the restriction folds a
// coarse cell without leaving the thread, in the reference's order.
//
// What bounds them: the f64 row arithmetic and the division were issued at
// 130 instructions a cell in the one-cell march (59% of the issue slots, DRAM
// at 30%).  Here it is 81; with 108 to 128 registers four blocks of four warps
// run per SM, and the latency of the rows' f64 chains bounds them (issue slots
// 35-48%, DRAM 27-48%).  On 128 x 128 x 256, one-cell march -> this, in us:
// direction + SpMV 38.4 -> 29.3, sweep 28.6 -> 25.6, with the prolongation 44.5
// -> 32.6, with the dots 44.4 -> 38.3, restriction 37.8 -> 25.8.  Every row is
// the same expression in the same order as in `stencil`, so the results are bit
// for bit those of the other kernels; only the order of the reductions follows
// the tile.
#pragma once

#include "efsi_march.cuh"

namespace efsi {

constexpr int kCK = 64;            // tile width along k (two cells per lane)
constexpr int kCWarps = 4;         // warps per block, two rows each
constexpr int kCJ = 2 * kCWarps;   // tile height along j
constexpr int kCThreads = 32 * kCWarps;

// Launch shape: `chunk` planes (even) per block, as march_cfg.
inline MarchCfg column_cfg(int nx, int ny, int nz, int slots) {
  const int tiles = ((nz + kCK - 1) / kCK) * ((ny + kCJ - 1) / kCJ);
  int nsplit = slots / tiles;
  if (nsplit < 1) nsplit = 1;
  int chunk = (nx + nsplit - 1) / nsplit;
  if (chunk < 2) chunk = 2;
  chunk += chunk & 1;
  MarchCfg c;
  c.chunk = chunk;
  c.grid = (unsigned)(tiles * ((nx + chunk - 1) / chunk));
  return c;
}

// A stage: NV value tiles of TV with halo, NR plain tiles of TR, the mask.
template <typename TV, int NV, typename TR, int NR, int kS>
struct ColumnStage {
  static constexpr int kPad = 16 / (int)sizeof(TV);
  static constexpr int kW = kCK + 2 * kPad;
  static constexpr int kVBytes = (kCJ + 2) * kW * (int)sizeof(TV);
  static constexpr int kRBytes = kCJ * kCK * (int)sizeof(TR);
  static constexpr int kMBytes = kCJ * kCK;
  static constexpr int kVStride = round128(kVBytes);
  static constexpr int kRStride = round128(kRBytes);
  static constexpr int kROff = NV * kVStride;
  static constexpr int kMOff = kROff + NR * kRStride;
  static constexpr int kStage = round128(kMOff + kMBytes);
  static constexpr int kBarOff = kS * kStage;
  static constexpr int kSmem = kBarOff + kS * 8 + 128;
};

struct ColumnGeom {
  int tx, ty;
  int j0, k0;
  int j, k;       // the thread's patch: rows j, j + 1, cells k, k + 1
  int ib, ie;
  bool act[2];    // row r lies inside the level (with both cells: the width is even)
  int64_t off[2]; // in-plane offset of (row r, k)
};

__device__ __forceinline__ bool column_geom(const LevelDev& L, int chunk, ColumnGeom& g) {
  const int ntk = (L.nz + kCK - 1) / kCK, ntj = (L.ny + kCJ - 1) / kCJ;
  int b = (int)blockIdx.x;
  const int tk = b % ntk;
  b /= ntk;
  const int tj = b % ntj;
  g.ib = (b / ntj) * chunk;
  g.ie = min(L.nx, g.ib + chunk);
  g.tx = (int)threadIdx.x;
  g.ty = (int)threadIdx.y;
  g.k0 = tk * kCK;
  g.j0 = tj * kCJ;
  g.k = g.k0 + 2 * g.tx;
  g.j = g.j0 + 2 * g.ty;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    g.act[r] = g.j + r < L.ny && g.k < L.nz;
    g.off[r] = (int64_t)(g.j + r) * L.nz + g.k;
  }
  return g.ib < g.ie;
}

// Two neighbouring cells of a tile.
template <typename T>
struct Pair;
template <>
struct Pair<double> {
  using type = double2;
};
template <>
struct Pair<float> {
  using type = float2;
};

template <typename TC>
struct Patch {
  TC v[2][2];  // [row][cell]
};

// Per-thread axis coefficients of the patch; CT is the arithmetic's type.
template <typename CT>
struct PatchCoef {
  CT ym[2], yp[2], zm[2], zp[2];
  unsigned edge[2];  // per row: faces on the domain's boundary, both cells (16 bits)
};

template <typename CT>
__device__ __forceinline__ PatchCoef<CT> patch_coef(const LevelDev& L, const ColumnGeom& g) {
  PatchCoef<CT> c;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int j = min(g.j + r, L.ny - 1), k = min(g.k + r, L.nz - 1);
    c.ym[r] = (CT)__ldg(L.cym + j);
    c.yp[r] = (CT)__ldg(L.cyp + j);
    c.zm[r] = (CT)__ldg(L.czm + k);
    c.zp[r] = (CT)__ldg(L.czp + k);
    unsigned e = 0;
    if (g.j + r == 0) e |= M_YM * 0x0101u;
    if (g.j + r == L.ny - 1) e |= M_YP * 0x0101u;
    if (g.k == 0) e |= M_ZM;
    if (g.k + 1 == L.nz - 1) e |= (unsigned)M_ZP << 8;
    // rows outside the level store nothing: they never ask for selection
    c.edge[r] = g.act[r] ? e : 0xFFFFu;
  }
  return c;
}

// The plane's six neighbour values of every cell of the patch.
template <typename TC>
struct Around {
  TC ym[2], yp[2];  // rows j - 1 and j + 2, cells k and k + 1
  TC zm[2], zp[2];  // cells k - 1 and k + 2, rows j and j + 1
};

// The march.  Op hooks, in order for every plane i:
//   op.centre(tiles, p, q): the patch of plane p (q: which of the pair's
//     planes, 2 for the plane after it), from its stage's value tiles;
//   op.plane(i, q, prev, cur, next, stage): the four cells of plane i;
// and op.pair(i) before the planes i and i + 1 (i even), op.first(p) before
// the centre of plane ib - 1.  Returns false in every thread if a stage did
// not land in time.
template <typename TV, int NV, typename TR, int NR, int kS, typename TC, class Op>
__device__ __forceinline__ bool column_march(const LevelDev& L, const ColumnGeom& g, const CUtensorMap* const (&mv)[NV],
                                             const CUtensorMap* const (&mr)[NR > 0 ? NR : 1], const CUtensorMap* mm,
                                             Op& op) {
  extern __shared__ unsigned char dsmem[];
  using Lay = ColumnStage<TV, NV, TR, NR, kS>;
  unsigned char* base = dsmem + ((128u - (smem_addr(dsmem) & 127u)) & 127u);
  uint64_t* bar = reinterpret_cast<uint64_t*>(base + Lay::kBarOff);
  const bool leader = g.tx == 0 && g.ty == 0;
  // plane p lives in stage (p - ib + 1) % kS, phase ((p - ib + 1) / kS) & 1;
  // the halo planes ib - 1 and ie carry only the value tiles
  auto issue = [&](int p) {
    const int s = (p - g.ib + 1) % kS;
    unsigned char* st = base + s * Lay::kStage;
    const bool interior = p >= g.ib && p < g.ie;
    mbar_expect_tx(&bar[s], NV * Lay::kVBytes + (interior ? NR * Lay::kRBytes + Lay::kMBytes : 0));
#pragma unroll
    for (int v = 0; v < NV; ++v) tma_load_3d(st + v * Lay::kVStride, mv[v], g.k0 - Lay::kPad, g.j0 - 1, p, &bar[s]);
    if (interior) {
#pragma unroll
      for (int r = 0; r < NR; ++r)
        tma_load_3d(st + Lay::kROff + r * Lay::kRStride, mr[r], g.k0, g.j0, p, &bar[s]);
      tma_load_3d(st + Lay::kMOff, mm, g.k0, g.j0, p, &bar[s]);
    }
  };
  if (leader) {
    for (int s = 0; s < kS; ++s) mbar_init(&bar[s], 1);
    mbar_fence_init();
  }
  __syncthreads();
  int issued = min(g.ie, g.ib - 2 + kS);  // last plane in flight
  if (leader)
    for (int p = g.ib - 1; p <= issued; ++p) issue(p);
  bool fail = false;
  auto stage = [&](int p) -> const unsigned char* { return base + ((p - g.ib + 1) % kS) * Lay::kStage; };
  auto wait = [&](int p) {
    if (!fail) fail = !mbar_wait(&bar[(p - g.ib + 1) % kS], (unsigned)(((p - g.ib + 1) / kS) & 1));
  };
  op.first(g.ib - 1);
  op.pair(g.ib);
  wait(g.ib - 1);
  Patch<TC> prev = op.centre(stage(g.ib - 1), g.ib - 1, -1);
  wait(g.ib);
  Patch<TC> cur = op.centre(stage(g.ib), g.ib, 0);
  for (int i = g.ib; i < g.ie; i += 2) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int p = i + q;
      if (p >= g.ie) break;
      wait(p + 1);
      if (__builtin_expect(!fail, 1)) {
        const Patch<TC> next = op.centre(stage(p + 1), p + 1, q + 1);
        op.plane(p, q, prev, cur, next, stage(p));
        prev = cur;
        cur = next;
      }
      if (q == 1 && p + 1 < g.ie) op.pair(p + 1);
      if (__syncthreads_or(fail)) {
        if (leader)  // let the copies in flight land before the block exits
          for (int c = p + 1; c <= issued; ++c)
            mbar_wait(&bar[(c - g.ib + 1) % kS], (unsigned)(((c - g.ib + 1) / kS) & 1));
        __syncthreads();
        return false;
      }
      // every plane up to p has been read by all threads: refill
      if (leader) {
        fence_proxy_async_smem();
        while (issued < min(g.ie, p + kS)) issue(++issued);
      }
    }
  }
  return true;
}

template <typename TV, typename TC, int kW, int kPad>
__device__ __forceinline__ Patch<TC> read_centre(const unsigned char* st, const ColumnGeom& g) {
  using V2 = typename Pair<TV>::type;
  const TV* at = reinterpret_cast<const TV*>(st) + (2 * g.ty + 1) * kW + kPad + 2 * g.tx;
  const V2 a = *reinterpret_cast<const V2*>(at), b = *reinterpret_cast<const V2*>(at + kW);
  return {{{(TC)a.x, (TC)a.y}, {(TC)b.x, (TC)b.y}}};
}

template <typename TV, typename TC, int kW, int kPad>
__device__ __forceinline__ Around<TC> read_around(const unsigned char* st, const ColumnGeom& g) {
  using V2 = typename Pair<TV>::type;
  const TV* at = reinterpret_cast<const TV*>(st) + (2 * g.ty + 1) * kW + kPad + 2 * g.tx;
  const V2 m = *reinterpret_cast<const V2*>(at - kW), p = *reinterpret_cast<const V2*>(at + 2 * kW);
  return {{(TC)m.x, (TC)m.y}, {(TC)p.x, (TC)p.y}, {(TC)at[-1], (TC)at[kW - 1]}, {(TC)at[2], (TC)at[kW + 2]}};
}

template <typename TR>
__device__ __forceinline__ Patch<double> read_plain(const unsigned char* tile, const ColumnGeom& g) {
  using R2 = typename Pair<TR>::type;
  const TR* at = reinterpret_cast<const TR*>(tile) + 2 * g.ty * kCK + 2 * g.tx;
  const R2 a = *reinterpret_cast<const R2*>(at), b = *reinterpret_cast<const R2*>(at + kCK);
  return {{{(double)a.x, (double)a.y}, {(double)b.x, (double)b.y}}};
}

__device__ __forceinline__ void read_masks(const unsigned char* tile, const ColumnGeom& g, unsigned (&m)[2]) {
  const uint8_t* at = tile + 2 * g.ty * kCK + 2 * g.tx;
  m[0] = *reinterpret_cast<const uint16_t*>(at);
  m[1] = *reinterpret_cast<const uint16_t*>(at + kCK);
}

constexpr unsigned kWhole = 0x7F7Fu;  // both cells fluid, all faces open

// Whether the warp's cells of this plane all have a whole stencil.
template <typename CT>
__device__ __forceinline__ bool whole_plane(const LevelDev& L, const PatchCoef<CT>& c, int i, const unsigned (&m)[2]) {
  unsigned edge = 0;
  if (i == 0) edge |= M_XM * 0x0101u;
  if (i == L.nx - 1) edge |= M_XP * 0x0101u;
  const unsigned a = m[0] | c.edge[0] | edge, b = m[1] | c.edge[1] | edge;
  // rows outside the level: 0xFFFF, with the solid bits masked out of the test
  const bool whole = (a & kWhole) == kWhole && (b & kWhole) == kWhole && (c.edge[0] == 0xFFFFu || !(m[0] & 0x8080u)) &&
                     (c.edge[1] == 0xFFFFu || !(m[1] & 0x8080u));
  return __all_sync(0xffffffffu, whole);
}

// Neighbour sum and denominator of cell (r, e) without selection; `stencil`'s
// expressions in its order.
template <typename CT>
__device__ __forceinline__ void stencil_whole(const PatchCoef<CT>& c, CT kxm, CT kxp, CT kx, int r, int e,
                                              const Patch<CT>& prev, const Patch<CT>& cur, const Patch<CT>& next,
                                              const Around<CT>& nb, CT& ns, CT& den) {
  const CT vym = r == 0 ? nb.ym[e] : cur.v[0][e], vyp = r == 0 ? cur.v[1][e] : nb.yp[e];
  const CT vzm = e == 0 ? nb.zm[r] : cur.v[r][0], vzp = e == 0 ? cur.v[r][1] : nb.zp[r];
  ns = kxm * prev.v[r][e];
  ns = fma(kxp, next.v[r][e], ns);
  ns = fma(c.ym[r], vym, ns);
  ns = fma(c.yp[r], vyp, ns);
  ns = fma(c.zm[e], vzm, ns);
  ns = fma(c.zp[e], vzp, ns);
  den = kx + c.ym[r];
  den += c.yp[r];
  den += c.zm[e];
  den += c.zp[e];
}

template <bool kAux>
__device__ __forceinline__ void stencil_select(const LevelDev& L, const PatchCoef<double>& c, double kxm, double kxp,
                                               int i, int r, int e, const ColumnGeom& g, int64_t cell, unsigned m,
                                               int outlet, const Patch<double>& prev, const Patch<double>& cur,
                                               const Patch<double>& next, const Around<double>& nb, double& ns,
                                               double& den) {
  const RowCoef rc = {c.ym[r], c.yp[r], c.zm[e], c.zp[e]};
  stencil_sel<kAux>(L, rc, kxm, kxp, i, g.j + r, g.k + e, cell, m, outlet, prev.v[r][e], next.v[r][e],
                    r == 0 ? nb.ym[e] : cur.v[0][e], r == 0 ? cur.v[1][e] : nb.yp[e],
                    e == 0 ? nb.zm[r] : cur.v[r][0], e == 0 ? cur.v[r][1] : nb.zp[r], ns, den);
}

template <bool kAux>
__device__ __forceinline__ void stencil_select(const LevelDev& L, const PatchCoef<float>& c, float kxm, float kxp,
                                               int i, int r, int e, const ColumnGeom& g, int64_t cell, unsigned m,
                                               int outlet, const Patch<float>& prev, const Patch<float>& cur,
                                               const Patch<float>& next, const Around<float>& nb, float& ns,
                                               float& den) {
  const RowCoef rc = {(double)c.ym[r], (double)c.yp[r], (double)c.zm[e], (double)c.zp[e]};
  stencil_sel32<kAux>(L, rc, kxm, kxp, i, g.j + r, g.k + e, cell, m, outlet, prev.v[r][e], next.v[r][e],
                      r == 0 ? nb.ym[e] : cur.v[0][e], r == 0 ? cur.v[1][e] : nb.yp[e],
                      e == 0 ? nb.zm[r] : cur.v[r][0], e == 0 ? cur.v[r][1] : nb.zp[r], ns, den);
}

// ---------------------------------------------------------------------------
// Sweeps (SweepOp of efsi_march.cuh: damped Jacobi, with the prolongation of
// the coarse iterate and the PCG's dots fused in).  TV is the iterate's type
// and the arithmetic's: double, or float for the mixed-precision V-cycle,
// whose result goes to `out64` when it is set.  The right-hand side is -r in
// f64.  With kRd the rows' reciprocal denominators come from a tile.
// ---------------------------------------------------------------------------
constexpr int kSweepStages = 5, kDotsStages = 3;

template <typename TV, bool kProlong, bool kAux, bool kDots>
struct ColumnSweep {
  static constexpr bool kF64 = sizeof(TV) == 8;
  // the reciprocals are kept for the f64 sweep that ends the V-cycle
  static constexpr bool kRd = kF64 && kDots;
  static constexpr int NR = 1 + (kDots ? 1 : 0) + (kRd ? 1 : 0);
  static constexpr int kS = kDots ? kDotsStages : kSweepStages;
  using Lay = ColumnStage<TV, 1, double, NR, kS>;

  const LevelDev& L;
  const ColumnGeom& g;
  TV* __restrict__ out;
  double* __restrict__ out64;
  int outlet;
  double omega;
  ProlongSrc pr;
  bool want_sum;
  PatchCoef<TV> pc;
  TV outz[2];          // the outlet's term of the denominator, per cell
  double wyz[2][2];    // widths of the patch along j and k
  double zsum, srz, sr, sdz, sd;
  // coarse values behind the patch and its four sides: of the pair's parent
  // plane, of the one after it, and the centre of the one before
  float cv[2][5], cbefore;
  int coff[5];

  __device__ __forceinline__ void init() {
    pc = patch_coef<TV>(L, g);
#pragma unroll
    for (int e = 0; e < 2; ++e) outz[e] = (outlet && g.k + e == 0) ? (TV)L.oz : (TV)0;
    zsum = srz = sr = sdz = sd = 0.0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      wyz[0][r] = (double)__ldg(L.wy + min(g.j + r, L.ny - 1));
      wyz[1][r] = (double)__ldg(L.wz + min(g.k + r, L.nz - 1));
    }
    if (kProlong) {
      auto par = [](int v, int n, int cn) { return min(min(max(v, 0), n - 1) / 2, cn - 1); };
      const int cj = par(g.j, L.ny, pr.cny), ck = par(g.k, L.nz, pr.cnz);
      coff[0] = cj * pr.cnz + ck;
      coff[1] = cj * pr.cnz + par(g.k - 1, L.nz, pr.cnz);
      coff[2] = cj * pr.cnz + par(g.k + 2, L.nz, pr.cnz);
      coff[3] = par(g.j - 1, L.ny, pr.cny) * pr.cnz + ck;
      coff[4] = par(g.j + 2, L.ny, pr.cny) * pr.cnz + ck;
    }
  }
  __device__ __forceinline__ const float* coarse_plane(int i) const {
    const int ci = min(min(max(i, 0), L.nx - 1) / 2, pr.cnx - 1);
    return pr.pc + (int64_t)ci * pr.cny * pr.cnz;
  }
  __device__ __forceinline__ float scaled(const float* plane, int q) const {
    return __fmul_rn(pr.scale, __ldg(plane + coff[q]));
  }
  __device__ __forceinline__ void first(int p) {
    if (!kProlong) return;
    cbefore = scaled(coarse_plane(p), 0);
    const float* c = coarse_plane(p + 1);
#pragma unroll
    for (int q = 0; q < 5; ++q) cv[1][q] = scaled(c, q);
  }
  __device__ __forceinline__ void pair(int i) {
    if (!kProlong) return;
    const float* c = coarse_plane(i + 2);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      cv[0][q] = cv[1][q];
      cv[1][q] = scaled(c, q);
    }
  }
  // p + s p_coarse in the level's precision
  __device__ __forceinline__ static TV corrected(TV v, float c) {
    if constexpr (kF64)
      return __dadd_rn(v, (double)c);
    else
      return __fadd_rn(v, c);
  }
  // Corrected whether or not the cell is fluid: neighbours behind open faces
  // are; a cell of neither kind reads its own value again below.
  __device__ __forceinline__ Patch<TV> centre(const unsigned char* st, int, int q) const {
    Patch<TV> p = read_centre<TV, TV, Lay::kW, Lay::kPad>(st, g);
    if (kProlong) {
      const float c = q < 0 ? cbefore : (q == 2 ? cv[1][0] : cv[0][0]);
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) p.v[r][e] = corrected(p.v[r][e], c);
    }
    return p;
  }

  __device__ __forceinline__ void plane(int i, int, const Patch<TV>& prev, const Patch<TV>& cur, const Patch<TV>& next,
                                        const unsigned char* st) {
    Around<TV> nb = read_around<TV, TV, Lay::kW, Lay::kPad>(st, g);
    if (kProlong) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        nb.zm[r] = corrected(nb.zm[r], cv[0][1]);
        nb.zp[r] = corrected(nb.zp[r], cv[0][2]);
        nb.ym[r] = corrected(nb.ym[r], cv[0][3]);
        nb.yp[r] = corrected(nb.yp[r], cv[0][4]);
      }
    }
    unsigned m[2];
    read_masks(st + Lay::kMOff, g, m);
    const Patch<double> rhs = read_plain<double>(st + Lay::kROff, g);
    Patch<double> dl, rd;
    if (kDots) dl = read_plain<double>(st + Lay::kROff + Lay::kRStride, g);
    if (kRd) rd = read_plain<double>(st + Lay::kROff + 2 * Lay::kRStride, g);
    const TV kxm = (TV)__ldg(L.cxm + i), kxp = (TV)__ldg(L.cxp + i);
    const TV om = (TV)omega;
    Patch<TV> res;
    bool whole = false;
    if (!kAux) whole = whole_plane(L, pc, i, m);
    if (whole) {
      const TV kx = kxm + kxp;
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          TV ns, den;
          stencil_whole(pc, kxm, kxp, kx, r, e, prev, cur, next, nb, ns, den);
          den += outz[e];
          const TV x0 = cur.v[r][e];
          TV jv;
          if constexpr (kRd)
            jv = (ns + rhs.v[r][e]) * rd.v[r][e];
          else
            jv = (ns + (TV)rhs.v[r][e]) / den;
          res.v[r][e] = x0 + om * (jv - x0);
        }
    } else {
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const unsigned mc = (m[r] >> (8 * e)) & 0xFFu;
          TV v = (TV)0;
          if (g.act[r] && !(mc & M_SOLID)) {
            const int64_t cell = (int64_t)i * L.ny * L.nz + g.off[r] + e;
            TV x0 = cur.v[r][e];
            if (kProlong && !(mc & M_FLUID))
              x0 = reinterpret_cast<const TV*>(st)[(2 * g.ty + 1 + r) * Lay::kW + Lay::kPad + 2 * g.tx + e];
            TV ns, den;
            stencil_select<kAux>(L, pc, kxm, kxp, i, r, e, g, cell, mc, outlet, prev, cur, next, nb, ns, den);
            if constexpr (kRd) {
              if (rd.v[r][e] > 0.0) v = x0 + om * ((ns + rhs.v[r][e]) * rd.v[r][e] - x0);
            } else {
              if (kAux) den += (TV)iface_at<double>(L, cell);
              if (den > (TV)0) v = x0 + om * ((ns + (TV)rhs.v[r][e]) / den - x0);
            }
          }
          res.v[r][e] = v;
        }
    }
    const int64_t pb = (int64_t)i * L.ny * L.nz;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (!g.act[r]) continue;
      const int64_t at = pb + g.off[r];
      if (kF64)
        *reinterpret_cast<double2*>(out + at) = make_double2((double)res.v[r][0], (double)res.v[r][1]);
      else if (out64 != nullptr)
        *reinterpret_cast<double2*>(out64 + at) = make_double2((double)res.v[r][0], (double)res.v[r][1]);
      else
        *reinterpret_cast<float2*>(out + at) = make_float2((float)res.v[r][0], (float)res.v[r][1]);
    }
    if (want_sum || kDots) {
      const double wx = (double)__ldg(L.wx + i);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const double wxy = wx * wyz[0][r];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (!g.act[r] || !((m[r] >> (8 * e)) & M_FLUID)) continue;
          const double vol = wxy * wyz[1][e], v = (double)res.v[r][e];
          zsum += v * vol;
          if (kDots) {
            srz += rhs.v[r][e] * v * vol;
            sr += rhs.v[r][e] * vol;
            sdz += v * dl.v[r][e] * vol;
            sd += dl.v[r][e] * vol;
          }
        }
      }
    }
  }
};

template <typename TV, bool kProlong, bool kAux, bool kDots>
__global__ void __launch_bounds__(kCThreads, 4)
    kc_sweep(LevelDev L, int chunk, const __grid_constant__ CUtensorMap map_p,
             const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_m,
             const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_rd,
             TV* __restrict__ out, double* __restrict__ out64, int outlet, double omega, ProlongSrc pr,
             double* partials, CgScalars* sc) {
  pdl_wait_early();
  using Op = ColumnSweep<TV, kProlong, kAux, kDots>;
  ColumnGeom g;
  const bool any = column_geom(L, chunk, g);
  Op op{L, g, out, out64, outlet, omega, pr, partials != nullptr};
  op.init();
  const CUtensorMap* const mv[1] = {&map_p};
  bool ok = true;
  if (any) {
    if constexpr (Op::NR == 1) {
      const CUtensorMap* const mr[1] = {&map_r};
      ok = column_march<TV, 1, double, 1, Op::kS, TV>(L, g, mv, mr, &map_m, op);
    } else if constexpr (Op::NR == 2) {
      const CUtensorMap* const mr[2] = {&map_r, &map_d};
      ok = column_march<TV, 1, double, 2, Op::kS, TV>(L, g, mv, mr, &map_m, op);
    } else {
      const CUtensorMap* const mr[3] = {&map_r, &map_d, &map_rd};
      ok = column_march<TV, 1, double, 3, Op::kS, TV>(L, g, mv, mr, &map_m, op);
    }
  }
  if (!ok) report_fault(sc);
  sweep_epilogue<kDots>(op, partials, sc);
}

// ---------------------------------------------------------------------------
// CG direction and SpMV (SpmvOp of efsi_march.cuh).
// ---------------------------------------------------------------------------
constexpr int kSpmvStages = 4;

template <bool kCopy, bool kAux>
struct ColumnSpmv {
  using Lay = ColumnStage<double, kCopy ? 1 : 2, double, 0, kSpmvStages>;
  const LevelDev& L;
  const ColumnGeom& g;
  double* __restrict__ d_new;
  double* __restrict__ Ad;
  int outlet;
  double beta, mz;
  int zproj;
  double part;
  PatchCoef<double> pc;
  double outz[2];
  double wyz[2][2];

  __device__ __forceinline__ void init() {
    pc = patch_coef<double>(L, g);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      outz[r] = (outlet && g.k + r == 0) ? L.oz : 0.0;
      wyz[0][r] = (double)__ldg(L.wy + min(g.j + r, L.ny - 1));
      wyz[1][r] = (double)__ldg(L.wz + min(g.k + r, L.nz - 1));
    }
  }
  __device__ __forceinline__ void first(int) {}
  __device__ __forceinline__ void pair(int) {}
  __device__ __forceinline__ double dir(double z, double d) const {
    if (zproj) z = z - mz;
    return kCopy ? z : z + beta * d;
  }
  __device__ __forceinline__ Patch<double> centre(const unsigned char* st, int, int) const {
    Patch<double> z = read_centre<double, double, Lay::kW, Lay::kPad>(st, g), d = z;
    if (!kCopy) d = read_centre<double, double, Lay::kW, Lay::kPad>(st + Lay::kVStride, g);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) z.v[r][e] = dir(z.v[r][e], d.v[r][e]);
    return z;
  }
  __device__ __forceinline__ void plane(int i, int, const Patch<double>& prev, const Patch<double>& cur,
                                        const Patch<double>& next, const unsigned char* st) {
    Around<double> nb = read_around<double, double, Lay::kW, Lay::kPad>(st, g), nd = nb;
    if (!kCopy) nd = read_around<double, double, Lay::kW, Lay::kPad>(st + Lay::kVStride, g);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      nb.ym[r] = dir(nb.ym[r], nd.ym[r]);
      nb.yp[r] = dir(nb.yp[r], nd.yp[r]);
      nb.zm[r] = dir(nb.zm[r], nd.zm[r]);
      nb.zp[r] = dir(nb.zp[r], nd.zp[r]);
    }
    unsigned m[2];
    read_masks(st + Lay::kMOff, g, m);
    const double kxm = __ldg(L.cxm + i), kxp = __ldg(L.cxp + i);
    const double wx = (double)__ldg(L.wx + i);
    const int64_t pb = (int64_t)i * L.ny * L.nz;
    bool whole = false;
    if (!kAux) whole = whole_plane(L, pc, i, m);
    Patch<double> o, x;
    if (whole) {
      const double kx = kxm + kxp;
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double ns, den;
          stencil_whole(pc, kxm, kxp, kx, r, e, prev, cur, next, nb, ns, den);
          den += outz[e];
          x.v[r][e] = cur.v[r][e];
          o.v[r][e] = (den + 0.0) * cur.v[r][e] - ns;
        }
    } else {
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const unsigned mc = (m[r] >> (8 * e)) & 0xFFu;
          double x0 = 0.0, v = 0.0;
          if (g.act[r] && !(mc & M_SOLID)) {
            const int64_t cell = pb + g.off[r] + e;
            x0 = cur.v[r][e];
            if (!(mc & M_FLUID) && zproj) {
              // z' = 0 off the fluid set
              const int at = (2 * g.ty + 1 + r) * Lay::kW + Lay::kPad + 2 * g.tx + e;
              x0 = kCopy ? 0.0 : 0.0 + beta * reinterpret_cast<const double*>(st + Lay::kVStride)[at];
            }
            double ns, den;
            stencil_select<kAux>(L, pc, kxm, kxp, i, r, e, g, cell, mc, outlet, prev, cur, next, nb, ns, den);
            v = (den + (kAux ? iface_at<double>(L, cell) : 0.0)) * x0 - ns;
          }
          x.v[r][e] = x0;
          o.v[r][e] = v;
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (!g.act[r]) continue;
      const int64_t at = pb + g.off[r];
      *reinterpret_cast<double2*>(d_new + at) = make_double2(x.v[r][0], x.v[r][1]);
      *reinterpret_cast<double2*>(Ad + at) = make_double2(o.v[r][0], o.v[r][1]);
      const double wxy = wx * wyz[0][r];
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if ((m[r] >> (8 * e)) & M_FLUID) part += x.v[r][e] * o.v[r][e] * (wxy * wyz[1][e]);
    }
  }
};

template <bool kCopy, bool kAux>
__global__ void __launch_bounds__(kCThreads, 4)
    kc_spmv_dir(LevelDev L, int chunk, const __grid_constant__ CUtensorMap map_z,
                const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_m,
                double* __restrict__ d_new, double* __restrict__ Ad, int outlet, double* partials, CgScalars* sc) {
  pdl_wait();
  ColumnGeom g;
  const bool any = column_geom(L, chunk, g);
  ColumnSpmv<kCopy, kAux> op{L, g, d_new, Ad, outlet, kCopy ? 0.0 : sc->beta, sc->mean_z, sc->zproj, 0.0};
  op.init();
  const CUtensorMap* const mr[1] = {nullptr};
  bool ok = true;
  if (any) {
    if constexpr (kCopy) {
      const CUtensorMap* const mv[1] = {&map_z};
      ok = column_march<double, 1, double, 0, kSpmvStages, double>(L, g, mv, mr, &map_m, op);
    } else {
      const CUtensorMap* const mv[2] = {&map_z, &map_d};
      ok = column_march<double, 2, double, 0, kSpmvStages, double>(L, g, mv, mr, &map_m, op);
    }
  }
  if (!ok) report_fault(sc);
  double v[1] = {op.part}, t[1];
  if (grid_sum<1>(v, partials, &sc->ticket, t)) {
    if (flat_tid() == 0) spmv_alpha(sc, t[0]);
  }
}

// ---------------------------------------------------------------------------
// Residual restriction (RestrictOp of efsi_march.cuh), with the coarse level's
// first sweep from a zero iterate when `cpa` is given.  TV is the iterate's
// storage type; the residual is formed in f64 and rounded to it.
// ---------------------------------------------------------------------------
template <typename TV, bool kAux>
struct ColumnRestrict {
  using Lay = ColumnStage<TV, 1, double, 1, kSweepStages>;
  const LevelDev& L;
  const ColumnGeom& g;
  int outlet;
  const LevelDev& C;  // the coarse level
  float* __restrict__ crhs;
  float* __restrict__ cpa;
  double omega;
  PatchCoef<double> pc;
  double outz[2];
  float wy[2], wz[2];
  float wres, free_vol;
  int solid;
  bool owner;  // the patch's coarse cell lies inside the coarse level
  int cj, ck;
  unsigned cm;  // the coarse cell's mask, loaded ahead

  __device__ __forceinline__ void init() {
    pc = patch_coef<double>(L, g);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      outz[r] = (outlet && g.k + r == 0) ? L.oz : 0.0;
      wy[r] = __ldg(L.wy + min(g.j + r, L.ny - 1));
      wz[r] = __ldg(L.wz + min(g.k + r, L.nz - 1));
    }
    wres = free_vol = 0.0f;
    solid = 0;
    cj = g.j >> 1;
    ck = g.k >> 1;
    owner = g.act[0] && cj < C.ny && ck < C.nz;
    cm = 0;
  }
  __device__ __forceinline__ void first(int) {}
  __device__ __forceinline__ void pair(int i) {
    if (cpa != nullptr && owner && (i >> 1) < C.nx) cm = __ldg(C.mask + cidx(i >> 1, cj, ck, C.ny, C.nz));
  }
  __device__ __forceinline__ Patch<double> centre(const unsigned char* st, int, int) const {
    return read_centre<TV, double, Lay::kW, Lay::kPad>(st, g);
  }
  __device__ __forceinline__ void plane(int i, int q, const Patch<double>& prev, const Patch<double>& cur,
                                        const Patch<double>& next, const unsigned char* st) {
    const Around<double> nb = read_around<TV, double, Lay::kW, Lay::kPad>(st, g);
    unsigned m[2];
    read_masks(st + Lay::kMOff, g, m);
    const Patch<double> rhs = read_plain<double>(st + Lay::kROff, g);
    const double kxm = __ldg(L.cxm + i), kxp = __ldg(L.cxp + i);
    const float wx = __ldg(L.wx + i);
    bool whole = false;
    if (!kAux) whole = whole_plane(L, pc, i, m);
    const double kx = kxm + kxp;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        double ns, den;
        bool is_solid = false;
        if (whole) {
          stencil_whole(pc, kxm, kxp, kx, r, e, prev, cur, next, nb, ns, den);
          den += outz[e];
        } else {
          const unsigned mc = (m[r] >> (8 * e)) & 0xFFu;
          is_solid = (mc & M_SOLID) != 0;
          ns = den = 0.0;
          if (g.act[r] && !is_solid) {
            const int64_t cell = (int64_t)i * L.ny * L.nz + g.off[r] + e;
            stencil_select<kAux>(L, pc, kxm, kxp, i, r, e, g, cell, mc, outlet, prev, cur, next, nb, ns, den);
            if (kAux) den += iface_at<TV>(L, cell);
          }
        }
        if (!g.act[r]) continue;  // odd heights: the last coarse row has one fine row
        if (is_solid) {
          solid += 1;
        } else {
          const double applied = ns - den * cur.v[r][e];
          const double res = (double)(TV)(-rhs.v[r][e] - applied);
          const float vol = __fmul_rn(__fmul_rn(wx, wy[r]), wz[e]);
          if (sizeof(TV) == 8)
            wres = (float)__dadd_rn((double)wres, __dmul_rn(res, (double)vol));
          else
            wres = __fadd_rn(wres, __fmul_rn((float)res, vol));
          free_vol = __fadd_rn(free_vol, vol);
        }
      }
    if (q == 1 || i == L.nx - 1) {
      const int ci = i >> 1;
      if (owner && ci < C.nx) {
        const int64_t cc = cidx(ci, cj, ck, C.ny, C.nz);
        const float v = solid > 0 ? 0.0f : __fdiv_rn(wres, fmaxf(free_vol, 1.0e-30f));
        crhs[cc] = v;
        if (cpa != nullptr) cpa[cc] = coarse_zero_sweep(C, cm, ci, cj, ck, cc, v, outlet, omega);
      }
      wres = free_vol = 0.0f;
      solid = 0;
    }
  }
};

template <typename TV, bool kAux>
__global__ void __launch_bounds__(kCThreads, 4)
    kc_restrict(LevelDev F, int chunk, const __grid_constant__ CUtensorMap map_p,
                const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_m, int outlet,
                LevelDev C, float* __restrict__ crhs, float* __restrict__ cpa, double omega, CgScalars* sc) {
  pdl_wait_early();
  ColumnGeom g;
  const bool any = column_geom(F, chunk, g);
  ColumnRestrict<TV, kAux> op{F, g, outlet, C, crhs, cpa, omega};
  op.init();
  const CUtensorMap* const mv[1] = {&map_p};
  const CUtensorMap* const mr[1] = {&map_r};
  if (any && !column_march<TV, 1, double, 1, kSweepStages, double>(F, g, mv, mr, &map_m, op)) report_fault(sc);
}

}  // namespace efsi
