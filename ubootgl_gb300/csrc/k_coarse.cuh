// The coarse end of the V-cycle in one block, every level's cells in
// registers while it is worked on (included by k_mg.cu after k_tile.cuh).
//
// A lane holds 4 columns of 2 rows, as in k_tile.cuh; a level of up to 4 n
// columns takes n = 4, 8, 16 or 32 lanes per row, so a warp holds 32 / n
// groups of two rows: 16 rows of 16 columns, 8 rows of 32, 4 rows of 64.
// Neighbours in a row and from group to group come by shuffle, only a warp's
// first and last row go through shared memory, and a level that fits one warp
// needs no barrier at all.  Between its visits a level's e and right-hand
// side lie in shared memory (rows of 4 n columns).  Edge cells of the
// reference's coarse levels are 0 and never updated; a solid cell and an edge
// cell have the factor 0.  The tolerance hierarchy's edge cells follow their
// inner neighbour (factor -1, as in k_tile.cuh).
//
// What bounds it: latency, a few hundred dependent instructions per visit.
// 64x32 and down: 11.7 us (ncu, cold).  The codes read level by level (a memory
// latency each) and the tolerance hierarchy's edges behind a uniform branch in
// every half sweep (132 against 80 cycles per half sweep of one warp) were 3 us
// more.  Before, with 4 columns x 2 rows per lane but always
// 32 lanes per row, all 32 warps and a block barrier per half sweep, 128x64 and
// down took 32 us: small levels waited for barriers of idle warps.  128x64 in
// the block instead of two smoothing launches (5 us each in a step): 43
// against 35 us per V-cycle of 256x128, hence the limit of 2048 cells.  The
// tolerance hierarchy's 65x33 in the block (17 warps) instead of two launches:
// 885 -> 871 us per step at 1024x512.  Its edge cells in registers: 374 -> 200
// cycles per half sweep of one warp.
#pragma once

namespace ubg {
namespace {
namespace coarse {

constexpr int kMaxLevels = 12;
// Warps of the block: the tolerance hierarchy's levels of 2^n + 1 columns and
// rows (65x33) take one group of rows more.
constexpr int warps_for(bool ext) { return ext ? 20 : 16; }
constexpr int kWarps = warps_for(true);
// Groups of four cells of all levels that a thread loads at most, and the block.
constexpr int kItems = 4;
constexpr int max_groups(bool ext) { return kItems * 32 * warps_for(ext); }

struct Level {
  int w, h, lsh, warps;   // lanes per row 1 << lsh; warps that hold its rows
  float hh, ihsq, rfac;
  int oe, of, oc;         // byte offsets of e, rhs (floats) and codes in shared memory
  const uint8_t *code;
  int code_pitch;
};
template <class S>
struct Args {
  int nlev;
  Level L[kMaxLevels];
  const S *rhs_top;
  int rhs_pitch;
  S *e_top;
  int e_pitch;
  float wsum[5], rwsum[5];
  int ext, ncoarse;  // tolerance hierarchy; sweeps on the coarsest level
};
// Lanes per row (log2) of a level of width w, and the warps for h rows.
inline int lane_shift(int w) { return w <= 16 ? 2 : (w <= 32 ? 3 : (w <= 64 ? 4 : 5)); }
inline int warps_of(int w, int h) {
  const int rows = 2 * (32 >> lane_shift(w));
  return (h + rows - 1) / rows;
}
// Groups of four cells of a level, and its bytes: e and rhs (16 per group) and
// codes (4), the next level's on a 16-byte boundary.
inline size_t groups_of(int w, int h) { return (size_t)h << lane_shift(w); }
inline size_t bytes_of(int w, int h) { return (36 * groups_of(w, h) + 15) / 16 * 16; }
// Shared memory before the levels: arguments (indexed by level, which in the
// parameter space would be a load from memory each time), exchanged rows of
// the warps and of one below and one above (zeros), restriction rows, table.
constexpr int kArgs = 0, kArgsBytes = 1024, kXch = kArgs + kArgsBytes,
              kRes = kXch + 2 * (kWarps + 2) * 512, kLut = kRes + (kWarps + 1) * 256,
              kLevels = (kLut + tile::kLutBytes + 15) / 16 * 16;

// A level's registers: two rows, columns (0, 2) and (1, 3).
struct Regs {
  float2 A[2], B[2], FA[2], FB[2];     // e and f h^2
  float2 sA[2], sB[2], cA[2], cB[2];   // factors (tile::scaled2)
  unsigned cw[2];
};
// Where a lane is in its level.
struct Place {
  int lsh, warps, wid, l, sub, groups;  // lane of the row, group of the warp
  int X, y;                             // first column and row
};

__device__ __forceinline__ float2 shfl2_up(float2 v, int d) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ float2 shfl2_down(float2 v, int d) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
// Barrier of the level's warps.
__device__ __forceinline__ void sync_level(int warps) {
  if (warps > 1)
    asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
  else
    __syncwarp();
}

// One half sweep (red or black).  MULTI: the level takes several warps.  EXT:
// the edge cells take their inner neighbour's value (follow) or keep theirs.
template <bool MULTI, bool CAREFUL, bool EXT, int RED>
__device__ __forceinline__ void half(Regs &q, const Place &pl, float2 *xch, const int w,
                                     const int h, const bool follow) {
  auto slot = [&](int buf, int wd, int lastrow) -> float2 & {
    return xch[((buf * (kWarps + 2) + 1 + wd) * 2 + lastrow) * 32];
  };
  const int n = 1 << pl.lsh, buf = RED ? 0 : 1;
  // pair updated in row 0: (1, 3) in a red half sweep, (0, 2) in a black one;
  // row 1 the other pair
  float2 below = shfl2_up(RED ? q.B[1] : q.A[1], n), above = shfl2_down(RED ? q.A[0] : q.B[0], n);
  if (pl.sub == 0) below = MULTI ? slot(buf, pl.wid - 1, 1) : make_float2(0.f, 0.f);
  if (pl.sub == pl.groups - 1) above = MULTI ? slot(buf, pl.wid + 1, 0) : make_float2(0.f, 0.f);
  float2 r2[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const bool onB = (r ^ RED) != 0;
    float2 W, E;
    if (onB) {
      W = q.A[r];
      E = make_float2(q.A[r].y, __shfl_down_sync(0xffffffffu, q.A[r].x, 1));
    } else {
      W = make_float2(__shfl_up_sync(0xffffffffu, q.B[r].y, 1), q.B[r].x);
      E = q.B[r];
    }
    const float2 S = r ? (onB ? q.B[0] : q.A[0]) : below, N = r ? above : (onB ? q.B[1] : q.A[1]);
    const float2 we = make_float2(W.x + E.x, W.y + E.y);
    float2 v = tile::add2(tile::add2(tile::add2(we, S), N), onB ? q.FB[r] : q.FA[r]);
    const float2 s = onB ? q.sB[r] : q.sA[r];
    if (EXT) {  // as in k_tile.cuh
      float2 t = make_float2(!onB && pl.X == 0 ? E.x : W.x, W.y);
      if (r == 0 && pl.y == 0) t = N;
      if (pl.y + r == h - 1) t = S;
      if (!follow) t = onB ? q.B[r] : q.A[r];
      if (__float_as_int(s.x) < 0) v.x = -t.x;
      if (__float_as_int(s.y) < 0) v.y = -t.y;
    }
    r2[r] = CAREFUL ? make_float2(tile::scaled_any(v.x, s.x), tile::scaled_any(v.y, s.y))
                    : tile::scaled2(v, s, onB ? q.cB[r] : q.cA[r]);
  }
  (RED ? q.B[0] : q.A[0]) = r2[0];
  (RED ? q.A[1] : q.B[1]) = r2[1];
  if (MULTI) {
    if (pl.sub == 0) slot(buf ^ 1, pl.wid, 0) = r2[0];
    if (pl.sub == pl.groups - 1) slot(buf ^ 1, pl.wid, 1) = r2[1];
    sync_level(pl.warps);
  }
}
template <bool MULTI, bool CAREFUL, bool EXT>
__device__ __forceinline__ void sweeps(Regs &q, const Place &pl, float2 *xch, const int w,
                                       const int h, const int n, const bool up) {
#pragma unroll 1
  for (int s = 0; s < n; s++) {
    half<MULTI, CAREFUL, EXT, 1>(q, pl, xch, w, h, up || s > 0);
    half<MULTI, CAREFUL, EXT, 0>(q, pl, xch, w, h, true);
  }
}

// One visit of level t by its warps: down (e = 0; sweeps, and unless it is the
// coarsest level residual and restriction to level t+1) or up (prolongation
// and correction from level t+1, sweeps).
template <class S, bool EXT>
__device__ __forceinline__ void visit(const Args<S> &a, const int t, const bool up,
                                      unsigned char *smem) {
  using St = Sto<S>;
  const Level &L = a.L[t];
  Place pl;
  const int lane = threadIdx.x & 31;
  pl.lsh = L.lsh;
  pl.warps = L.warps;
  pl.wid = threadIdx.x >> 5;
  pl.l = lane & ((1 << pl.lsh) - 1);
  pl.sub = lane >> pl.lsh;
  pl.groups = 32 >> pl.lsh;
  pl.X = 4 * pl.l;
  pl.y = 2 * (pl.wid * pl.groups + pl.sub);
  const int w = L.w, h = L.h, X = pl.X, y = pl.y, n = 1 << pl.lsh, stride = 4 * n;
  const bool last = t == a.nlev - 1;
  float *const e = reinterpret_cast<float *>(smem + L.oe) + y * stride + X;
  const float *const f = reinterpret_cast<const float *>(smem + L.of) + y * stride + X;
  const uint8_t *const code = smem + L.oc + y * stride + X;
  float2 *const xch = reinterpret_cast<float2 *>(smem + kXch) + pl.l;
  float2 *const res = reinterpret_cast<float2 *>(smem + kRes) + pl.l;
  const float2 *const lut = reinterpret_cast<const float2 *>(smem + kLut);
  auto slot = [&](int buf, int wd, int lastrow) -> float2 & {
    return xch[((buf * (kWarps + 2) + 1 + wd) * 2 + lastrow) * 32];
  };
  Regs q;
  unsigned inmask = 0u;
#pragma unroll
  for (int b = 0; b < 4; b++) inmask |= X + b >= 1 && X + b < w - 1 ? 0xffu << (8 * b) : 0u;
  float u[2][4];  // the correction of the two rows
  if (up) {
    // coarse rows y/2 and y/2 + 1 (columns past the coarse width hold 0; the
    // last row of an odd height lies over no coarse row)
    const Level &C = a.L[t + 1];
    const int cs = 4 << C.lsh, cx = X >> 1, cy = y >> 1;
    const float *ec = reinterpret_cast<const float *>(smem + C.oe) + cy * cs + cx;
    const uint8_t *cc = smem + C.oc + cy * cs + cx;
    float2 v0 = make_float2(0.f, 0.f), v1 = v0;
    unsigned g0 = 0u, g1 = 0u;
    if (cx < cs && cy < C.h) {
      v0 = *reinterpret_cast<const float2 *>(ec);
      g0 = *reinterpret_cast<const unsigned short *>(cc) & 0x0101u;
      if (cy + 1 < C.h) {
        v1 = *reinterpret_cast<const float2 *>(ec + cs);
        g1 = *reinterpret_cast<const unsigned short *>(cc + cs) & 0x0101u;
      }
    }
    const float e3[3] = {v0.x, v0.y, __shfl_down_sync(0xffffffffu, v0.x, 1)};
    const float f3[3] = {v1.x, v1.y, __shfl_down_sync(0xffffffffu, v1.x, 1)};
    g0 |= (__shfl_down_sync(0xffffffffu, g0, 1) & 1u) << 16;
    g1 |= (__shfl_down_sync(0xffffffffu, g1, 1) & 1u) << 16;
    tile::prolongate2(e3, f3, g0, g1, lut, u);
    if (!EXT) {  // no coarse cell beyond
#pragma unroll
      for (int b = 0; b < 4; b++) {
        if ((b & 1) && X + b >= w - 2) u[0][b] = u[1][b] = 0.0f;
        if (y + 1 >= h - 2) u[1][b] = 0.0f;
      }
    }
  }
  const float hh = L.hh;
  float2 sq = make_float2(0.f, 0.f);
  unsigned ef[2] = {0u, 0u};  // flags of the edge cells (EXT)
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int yy = y + r;
    float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f), fv = p4;
    unsigned c = 0u;   // smoothed cells' codes, 0 elsewhere
    unsigned ci = 0u;  // the table's index of each factor
    if (yy < h) {
      fv = *reinterpret_cast<const float4 *>(f + r * stride);
      if (up) p4 = *reinterpret_cast<const float4 *>(e + r * stride);
      const unsigned raw = *reinterpret_cast<const unsigned *>(code + r * stride);
      const unsigned in = yy >= 1 && yy < h - 1 ? inmask : 0u;
      c = raw & in;
      ci = c & 0x1f1f1f1fu;
      if (EXT) ci |= ~in & ((raw & 0x01010101u) | 0x20202020u);
      if (EXT) ef[r] = raw & 0x01010101u & ~in;
    }
    float p[4] = {p4.x, p4.y, p4.z, p4.w};
    float F[4] = {fv.x * hh * hh, fv.y * hh * hh, fv.z * hh * hh, fv.w * hh * hh};
    float s[4];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      if (up) p[b] = p[b] + u[r][b];
      if (!((c >> (8 * b)) & C_CENTER)) p[b] = F[b] = 0.0f;
      s[b] = reinterpret_cast<const float *>(lut)[(ci >> (8 * b)) & 0x3fu];
    }
    q.A[r] = make_float2(p[0], p[2]);
    q.B[r] = make_float2(p[1], p[3]);
    q.FA[r] = make_float2(F[0], F[2]);
    q.FB[r] = make_float2(F[1], F[3]);
    q.sA[r] = make_float2(s[0], s[2]);
    q.sB[r] = make_float2(s[1], s[3]);
    q.cA[r] = tile::third2(q.sA[r]);
    q.cB[r] = tile::third2(q.sB[r]);
    q.cw[r] = c;
    sq = f2_fma(q.FB[r], q.FB[r], f2_fma(q.FA[r], q.FA[r], sq));
    sq = f2_fma(q.B[r], q.B[r], f2_fma(q.A[r], q.A[r], sq));
  }
  if (EXT && up) {  // edge cells: their inner neighbours' corrected values
    const int pe = w - 1 - X;
    auto flag = [&](int r, int b, float v) { return (ef[r] >> (8 * b)) & 1u ? v : 0.0f; };
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const float left = __shfl_up_sync(0xffffffffu, q.B[r].y, 1);
      if (X == 0) q.A[r].x = flag(r, 0, q.B[r].x);
      if (pe == 0) q.A[r].x = flag(r, 0, left);
      if (pe == 1) q.B[r].x = flag(r, 1, q.A[r].x);
      if (pe == 2) q.A[r].y = flag(r, 2, q.B[r].x);
      if (pe == 3) q.B[r].y = flag(r, 3, q.A[r].y);
    }
    // rows 0 and h-1 (of the row below for a lane's first row, by shuffle; a
    // warp's first row is written by the warp below it, further down)
    const float2 bA = shfl2_up(q.A[1], n), bB = shfl2_up(q.B[1], n);
    auto row = [&](int r, float2 a, float2 b) {
      q.A[r] = make_float2(flag(r, 0, a.x), flag(r, 2, a.y));
      q.B[r] = make_float2(flag(r, 1, b.x), flag(r, 3, b.y));
    };
    if (y == 0) row(0, q.A[1], q.B[1]);
    if (y == h - 1) row(0, bA, bB);
    if (y + 1 == h - 1) row(1, q.A[0], q.B[0]);
  }
  // sums that may not stay finite (false for infinities and NaNs too): a warp
  // alone decides for itself, several agree through shared memory
  bool careful = __any_sync(0xffffffffu, !(sq.x + sq.y < tile::kBigSq<float>)) != 0;
  const bool multi = pl.warps > 1;
  if (multi) {
    const bool init = EXT && up;
    if (pl.sub == 0 && !(init && pl.wid > 0 && y == h - 1)) slot(0, pl.wid, 0) = q.A[0];
    if (init && pl.sub == pl.groups - 1 && pl.wid < pl.warps - 1 && y + 2 == h - 1)
      slot(0, pl.wid + 1, 0) = make_float2((q.cw[1] & C_N) ? q.A[1].x : 0.0f,
                                           ((q.cw[1] >> 16) & C_N) ? q.A[1].y : 0.0f);
    if (pl.sub == pl.groups - 1) slot(0, pl.wid, 1) = q.B[1];
    // the row above the last warp's: zeros
    if (pl.wid == pl.warps - 1 && pl.sub == 0)
      slot(0, pl.wid + 1, 0) = slot(1, pl.wid + 1, 0) = make_float2(0.f, 0.f);
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
                 "barrier.cta.red.or.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(any)
                 : "r"((int)careful), "r"(32 * pl.warps)
                 : "memory");
    careful = any != 0;
  }
  const int ns = last ? (EXT ? a.ncoarse : 5) : 3;
  if (careful) {
    if (multi)
      sweeps<true, true, EXT>(q, pl, xch, w, h, ns, up);
    else
      sweeps<false, true, EXT>(q, pl, xch, w, h, ns, up);
  } else if (multi) {
    sweeps<true, false, EXT>(q, pl, xch, w, h, ns, up);
  } else {
    sweeps<false, false, EXT>(q, pl, xch, w, h, ns, up);
  }

  // ---- e to shared memory, or the result to the top level's array.  Edge
  // cells: 0, or their inner neighbour's value (corners: the diagonal one's)
  const bool top = t == 0 && (up || last);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int yy = y + r;
    float o[4] = {q.A[r].x, q.B[r].x, q.A[r].y, q.B[r].y};
    if (EXT) {
      const float left = __shfl_up_sync(0xffffffffu, q.B[r].y, 1);
      const float inner[4] = {left, o[0], o[1], o[2]};
      if (X == 0) o[0] = o[1];
#pragma unroll
      for (int b = 0; b < 4; b++)
        if (X + b == w - 1) o[b] = inner[b];
    }
    auto put = [&](int ye) {
      if (ye >= h) return;
      if (top) {
        S *dst = a.e_top + (size_t)ye * a.e_pitch + X;
        if (X + 3 < w) {
          St::st4(dst, make_float4(o[0], o[1], o[2], o[3]));
        } else {
#pragma unroll
          for (int b = 0; b < 3; b++)
            if (X + b < w) dst[b] = St::fromf(o[b]);
        }
      } else {
        *reinterpret_cast<float4 *>(e + (ye - y) * stride) = make_float4(o[0], o[1], o[2], o[3]);
      }
    };
    if (!EXT || (yy >= 1 && yy < h - 1)) put(yy);
    if (EXT && yy == 1) put(0);
    if (EXT && yy == h - 2) put(h - 1);
  }
  if (up || last) return;

  // ---- residual (calculateResidualField, pressure_solver.cpp:91-116) and
  // restriction (pressure_solver.cpp:118-132) to level t+1
  float2 bA = shfl2_up(q.A[1], n), bB = shfl2_up(q.B[1], n);
  float2 tA = shfl2_down(q.A[0], n), tB = shfl2_down(q.B[0], n);
  if (multi && pl.sub == 0) {
    bA = slot(1, pl.wid - 1, 1);
    bB = slot(0, pl.wid - 1, 1);
  }
  if (multi && pl.sub == pl.groups - 1) {
    tA = slot(0, pl.wid + 1, 0);
    tB = slot(1, pl.wid + 1, 0);
  }
  float2 tt[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const float2 SA = r ? q.A[0] : bA, SB = r ? q.B[0] : bB;
    const float2 NA = r ? tA : q.A[1], NB = r ? tB : q.B[1];
    const float l = __shfl_up_sync(0xffffffffu, q.B[r].y, 1);
    const float rr = __shfl_down_sync(0xffffffffu, q.A[r].x, 1);
    float4 fv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (y + r < h) fv = *reinterpret_cast<const float4 *>(f + r * stride);
    const float C4[4] = {q.A[r].x, q.B[r].x, q.A[r].y, q.B[r].y};
    const float F4[4] = {fv.x, fv.y, fv.z, fv.w};
    float W4[4] = {l, q.A[r].x, q.B[r].x, q.A[r].y}, E4[4] = {q.B[r].x, q.A[r].y, q.B[r].y, rr};
    float S4[4] = {SA.x, SB.x, SA.y, SB.y}, N4[4] = {NA.x, NB.x, NA.y, NB.y};
    if (EXT) {  // the edge cells have this cell's value
#pragma unroll
      for (int b = 0; b < 4; b++) {
        if (X + b == 1) W4[b] = C4[b];
        if (X + b == w - 2) E4[b] = C4[b];
        if (y + r == 1) S4[b] = C4[b];
        if (y + r == h - 2) N4[b] = C4[b];
      }
    }
    float d[4];
    tile::residual4(q.cw[r], C4, W4, E4, S4, N4, F4, L.ihsq, d);
    const float dl = __shfl_up_sync(0xffffffffu, d[3], 1);
    // 1-2-1 or 2-4-2 (products by powers of two are exact)
    if (r)
      tt[r] = make_float2(__fmaf_rn(d[0], 2.0f, dl) + d[1], __fmaf_rn(d[2], 2.0f, d[1]) + d[3]);
    else
      tt[r] = make_float2(__fmaf_rn(d[1], 2.0f, __fmaf_rn(d[0], 4.0f, dl * 2.0f)),
                          __fmaf_rn(d[3], 2.0f, __fmaf_rn(d[2], 4.0f, d[1] * 2.0f)));
  }
  float2 tb = shfl2_up(tt[1], n);
  if (multi) {
    if (pl.sub == pl.groups - 1) res[(pl.wid + 1) * 32] = tt[1];
    sync_level(pl.warps);
    if (pl.sub == 0) tb = res[pl.wid * 32];
  }
  const Level &C = a.L[t + 1];
  const int c0 = X >> 1, cs = 4 << C.lsh, Y = y >> 1;
  float v0 = ((tb.x + tt[0].x) + tt[1].x) * L.rfac;
  float v1 = ((tb.y + tt[0].y) + tt[1].y) * L.rfac;
  const bool yz = Y == 0 || Y >= C.h - 1;
  if (yz || c0 == 0 || c0 >= C.w - 1) v0 = 0.0f;
  if (yz || c0 + 1 >= C.w - 1) v1 = 0.0f;
  if (Y < C.h && c0 < cs)
    *reinterpret_cast<float2 *>(reinterpret_cast<float *>(smem + C.of) + Y * cs + c0) =
        make_float2(v0, v1);
}

// What needs no other kernel's results: arguments and zero rows to shared
// memory.
template <class S>
__device__ __forceinline__ void init(const Args<S> &args, unsigned char *smem) {
  static_assert(sizeof(Args<S>) <= kArgsBytes && sizeof(Args<S>) % 4 == 0, "arguments");
  if (threadIdx.x < sizeof(Args<S>) / 4)
    reinterpret_cast<unsigned *>(smem + kArgs)[threadIdx.x] =
        reinterpret_cast<const unsigned *>(&args)[threadIdx.x];
  // the rows below the first warp's: zeros
  float2 *const xch = reinterpret_cast<float2 *>(smem + kXch);
  if (threadIdx.x < 128) xch[(threadIdx.x >> 6) * (kWarps + 2) * 64 + (threadIdx.x & 63)] = make_float2(0.f, 0.f);
  if (threadIdx.x < 32) reinterpret_cast<float2 *>(smem + kRes)[threadIdx.x] = make_float2(0.f, 0.f);
  __syncthreads();
}

template <class S, bool EXT>
__device__ __forceinline__ void run(unsigned char *smem) {
  using St = Sto<S>;
  constexpr int NT = 32 * warps_for(EXT);
  const Args<S> &a = *reinterpret_cast<const Args<S> *>(smem + kArgs);
  // Codes of every level, the top level's right-hand side (columns past the
  // width: 0).  The levels' groups of four cells are numbered through, at
  // most kItems per thread (max_groups: 16 x 256 cells and the levels below are
  // 1792 groups of the reference's hierarchy's 2048, 14 x 292 cells 2052 of the
  // tolerance hierarchy's 2560), and all their loads are in flight together.
  const uint8_t *src[kItems];
  unsigned mask[kItems], dst[kItems], c[kItems];
  int left[kItems];
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    left[k] = threadIdx.x + NT * k;
    src[k] = nullptr;
    mask[k] = dst[k] = c[k] = 0u;
  }
  const Level &T = a.L[0];
  const int nt = T.h << T.lsh, n1 = (1 << T.lsh) - 1;
#pragma unroll 1
  for (int t = 0; t < a.nlev; t++) {
    const Level &L = a.L[t];
    const int n = L.h << L.lsh;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
      const int i = left[k], X = 4 * (i & ((1 << L.lsh) - 1));
      left[k] -= n;
      if (i < 0 || i >= n) continue;
      dst[k] = L.oc + 4 * i;
      if (X >= L.w) continue;
      src[k] = L.code + (size_t)(i >> L.lsh) * L.code_pitch + X;
      mask[k] = 0xffffffffu >> (8 * max(0, X + 4 - L.w));
    }
  }
  float4 fv[kItems];
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    if (src[k]) c[k] = __ldg(reinterpret_cast<const unsigned *>(src[k])) & mask[k];
    const int i = threadIdx.x + NT * k, X = 4 * (i & n1);
    fv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < nt && X < T.w) fv[k] = St::ldg4(a.rhs_top + (size_t)(i >> T.lsh) * a.rhs_pitch + X);
  }
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    if (dst[k]) *reinterpret_cast<unsigned *>(smem + dst[k]) = c[k];
    const int i = threadIdx.x + NT * k;
    if (i < nt) *reinterpret_cast<float4 *>(smem + T.of + 16 * i) = fv[k];
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5;
#pragma unroll 1
  for (int v = 0; v < 2 * a.nlev - 1; v++) {
    const bool up = v >= a.nlev;
    const int t = up ? 2 * a.nlev - 2 - v : v;
    if (v == 2 * a.nlev - 2) griddep_launch();
    if (wid < a.L[t].warps) visit<S, EXT>(a, t, up, smem);
    // the next level's warps read what these wrote
    __syncthreads();
  }
}

}  // namespace coarse
}  // namespace
}  // namespace ubg
