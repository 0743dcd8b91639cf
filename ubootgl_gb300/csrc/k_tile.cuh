// The smoothing launch of the multigrid on tiles held in registers (included
// by k_mg.cu, which defines the stencil codes and the launch arguments).
//
// A block of NW warps owns a region of 128 columns x NW * R rows: a warp R
// consecutive rows, a lane 4 columns of them, as the column pairs (0, 2) and
// (1, 3).  p and f h^2 stay in registers over the three red-black sweeps: the
// neighbours in a row come from the next lane by shuffle, those above and
// below are the lane's own registers, and only a warp's first and last row go
// through shared memory, one barrier per half sweep.  A half sweep updates
// one pair of every row, so its sums are packed FP32 additions.
//
// A solid cell holds 0, so a sum needs no flag tests: the flags only decide
// what it is divided by.  A warp whose cells and all their neighbours are
// fluid takes val / 4; any other reads a factor per cell (1/n) from shared
// memory, where the block put them when it loaded the codes.
//
// After half sweep i, the cells within i of the region's edge are no longer
// exact, so regions overlap by 16 columns and rows and store what is 8 or
// more inside (all of it at the domain's edge).
//
// What bounds it: instruction issue and the FP32 pipe on large levels, the
// latency of loads, six barriers and one pass through the code on small ones.
// Against tiles in shared memory (red/black-split, 112 x 50 and 48 x 16
// cells), ncu: level 0 of 4096x2048 52.7 us (88.4) and 25.1 M warp instructions
// with the residual, 50.8 us (96.6) and 25.3 M with the prolongation; level 1
// (2048x1024) 18.5 us (34.3, 39.5), level 2 9 us (18.5), smaller ones 7 us.  Edge cells in the registers instead of neighbours rebuilt from codes
// and positions: 5900 -> 2260 cycles for an edge warp's six half sweeps (2000
// for others), 83 -> 78 us per step of 256x128.  Bounds checks outside the
// blocks that need them, the packed magnitude check and W + E as scalar
// additions (no register moves) were 2 us and a fifth of the instructions, f
// kept in shared memory for the residual and one factor per cell another 2
// (4096x2048 steps 660 -> 647 us).  Regions of 8 rows per warp (8 warps), and of
// 128 x 32 cells, are slower there (58-60, 65 us).
#pragma once

namespace ubg {
namespace {
namespace tile {

constexpr int kHalo = 8;
constexpr int kWarps = 16;
constexpr float kThird = 1.0f / 3.0f;
constexpr unsigned kFull = 0x1f1f1f1fu;

// Regions of n cells each with an overlap of 2 * kHalo that cover c cells.
__host__ __device__ constexpr int regions(int c, int n) {
  return c <= n ? 1 : (c - 2 * kHalo + n - 2 * kHalo - 1) / (n - 2 * kHalo);
}
// Shared memory: f and factors of each row (512 bytes each), exchanged rows of each warp
// (and of one below and one above: zeros), restriction rows, table of factors
// by code and of the prolongation's weight sums.
constexpr int kLutBytes = 64 * 4 + 5 * 8;
template <int R, int NW>
struct Mem {
  static constexpr int fac = 0, xch = fac + R * NW * 1024, res = xch + 2 * (NW + 2) * 512,
                       lut = res + (NW + 1) * 256, bytes = lut + kLutBytes;
};

// Two operations in one instruction, each lane rounded as its scalar form.
// No product is added by add2: ptxas may fuse a packed product with a packed
// addition.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// Asynchronous copy of B bytes to shared memory (zeros unless ok).
template <int B>
__device__ __forceinline__ void copy_async(void *dst, const void *src, bool ok) {
  const int n = ok ? B : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(B), "r"(n)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <class S>
__device__ __forceinline__ float rnd(float v) {
  if constexpr (std::is_same<S, float>::value)
    return v;
  else
    return Sto<S>::tof(Sto<S>::fromf(v));
}
template <class S>
__device__ __forceinline__ float2 rnd2(float2 v) {
  return make_float2(rnd<S>(v.x), rnd<S>(v.y));
}

// val / n of a pair: s = 1/n (the rounded third for n = 3; 0 for a solid cell
// or one without fluid neighbours).  n = 1, 2, 4 are exact products; n = 3 is
// Markstein's correction, whose remainder v - 3 q is exact for every finite v,
// subnormal results included (3 has two bits).  For finite sums only: 0 *
// infinity would be NaN.  c: third2(s).
__device__ __forceinline__ float2 third2(float2 s) {
  return make_float2(s.x == kThird ? kThird : 0.0f, s.y == kThird ? kThird : 0.0f);
}
__device__ __forceinline__ float2 scaled2(float2 v, float2 s, float2 c) {
  const float2 q = f2_mul(v, s);
  return f2_fma(f2_fma(q, f2(-3.0f), v), c, q);
}
// The same for any v (a solid cell is 0 whatever its sum).
__device__ __forceinline__ float scaled_any(float v, float s) {
  const float q = v * s;
  const float q3 = __fmaf_rn(__fmaf_rn(-q, 3.0f, v), s, q);
  const float n = (s == kThird && fabsf(v) < __int_as_float(0x7f800000)) ? q3 : q;
  return s != 0.0f ? n : 0.0f;
}
// Bound of the sum of squares of what a lane holds, p and kWeightF f h^2, under
// which the sweeps stay finite.  A half sweep gives at most the largest p plus
// the largest f h^2, rounded to S: in FP32 and BF16 values below 2^60 stay below
// 2^66 over the 32 half sweeps of the tolerance hierarchy's coarsest level; in
// FP16 p < 2^15 and f h^2 < 2^12 stay below 57600 over a launch's six, of 65504.
template <class S>
constexpr bool kIsHalf = std::is_same<S, __half>::value;
template <class S>
constexpr float kBigSq = kIsHalf<S> ? 0x1p+30f : 0x1p+120f;
template <class S>
constexpr float kWeightF = kIsHalf<S> ? 8.0f : 1.0f;

// Fills the table: factors by code, 32 + flag for a cell on the domain's
// edge; then the weight sums of the prolongation and their reciprocals.
__device__ __forceinline__ void fill_lut(float2 *lut, int i, const float *wsum,
                                         const float *rwsum) {
  if (i < 64) {
    const int n = __popc((i >> 1) & 15);
    float s = n == 4 ? 0.25f : (n == 3 ? kThird : (n == 2 ? 0.5f : (n == 1 ? 1.0f : 0.0f)));
    if (!(i & (int)C_CENTER)) s = 0.0f;
    if (i >= 32) s = i & (int)C_CENTER ? -1.0f : -0.0f;
    reinterpret_cast<float *>(lut)[i] = s;
  } else if (i < 69) {
    lut[i - 32] = make_float2(wsum[i - 64], rwsum[i - 64]);
  }
}

// prolongate (pressure_solver.cpp:134-172) onto two rows of a lane's four
// columns: coarse columns X/2, X/2 + 1 and X/2 + 2 of the coarse row below
// (e, flags g, one byte each) and the next one (f, g1); the first row lies
// over the coarse row, the second between the two.  u[row][column].
__device__ __forceinline__ void prolongate2(const float (&e)[3], const float (&f)[3], unsigned g,
                                            unsigned g1, const float2 *lut, float (&u)[2][4]) {
  const float v[6] = {e[0] + e[1],
                      e[1] + e[2],
                      e[0] + f[0],
                      ((e[0] + f[1]) + e[1]) + f[0],
                      e[1] + f[1],
                      ((e[1] + f[2]) + e[2]) + f[1]};
  float2 d[6];
  if (__all_sync(0xffffffffu, (g & g1) == 0x010101u)) {
    const float2 d2 = lut[34], d4 = lut[36];
#pragma unroll
    for (int i = 0; i < 6; i++) d[i] = i == 3 || i == 5 ? d4 : d2;
  } else {
    const unsigned t = g + g1;  // flag sums of the column pairs, a byte each
    d[0] = lut[32 + (g & 1u) + ((g >> 8) & 1u)];
    d[1] = lut[32 + ((g >> 8) & 1u) + (g >> 16)];
    d[2] = lut[32 + (t & 0xffu)];
    d[3] = lut[32 + (t & 0xffu) + ((t >> 8) & 0xffu)];
    d[4] = lut[32 + ((t >> 8) & 0xffu)];
    d[5] = lut[32 + ((t >> 8) & 0xffu) + (t >> 16)];
  }
  float q[6];
  unsigned lo = ~0u;
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 6; i++) {  // div_rn's correction
    const float q0 = v[i] * d[i].y;
    q[i] = __fmaf_rn(__fmaf_rn(-q0, d[i].x, v[i]), d[i].y, q0);
    lo = min(lo, div_key(v[i]));
    m = m + fabsf(v[i]);
  }
  // sums the correction is not exact for (zeros are fine)
  if (!__all_sync(0xffffffffu, lo >= kDivKeyLo && m <= 0x1p+100f)) {
#pragma unroll
    for (int i = 0; i < 6; i++) q[i] = div_rn(v[i], d[i].x, d[i].y);
  }
  u[0][0] = e[0];
  u[0][1] = q[0];
  u[0][2] = e[1];
  u[0][3] = q[1];
#pragma unroll
  for (int b = 0; b < 4; b++) u[1][b] = q[2 + b];
}

// Residuals (calculateResidualField, pressure_solver.cpp:91-116) of a lane's
// four cells with codes c (center bit clear: 0): values C, W, E, S, N, right
// hand side F.
__device__ __forceinline__ void residual4(unsigned c, const float (&C)[4], const float (&W)[4],
                                          const float (&E)[4], const float (&S)[4],
                                          const float (&N)[4], const float (&F)[4], float ihsq,
                                          float (&q)[4]) {
#pragma unroll
  for (int b = 0; b < 4; b++) {
    const unsigned k = c >> (8 * b);
    const float v = (((((k & C_W) ? W[b] : C[b]) + ((k & C_E) ? E[b] : C[b])) +
                      ((k & C_S) ? S[b] : C[b])) +
                     ((k & C_N) ? N[b] : C[b])) +
                    -4.0f * C[b];
    q[b] = (k & C_CENTER) ? F[b] + v * ihsq : 0.0f;
  }
}

// One region of the level: columns from 112 * sx, rows from (NW * R - 16) * sy.
// PRE: residual and restriction (a.rc); else prolongation and correction (a.ec)
// first.  Red points are those with x + y odd; even rows
// hold them in the pair (1, 3).
template <class S, class SC, bool EXT, bool PRE, int R, int NW>
__device__ __forceinline__ void run(const MgArgsT<S, SC> &a, const int region,
                                    unsigned char *smem) {
  static_assert(R % 2 == 0, "row parity");
  using M = Mem<R, NW>;
  using St = Sto<S>;
  using Sc = Sto<SC>;
  constexpr int RY = R * NW;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = a.w, h = a.h;
  const size_t P = (size_t)a.pitch;
  const int nsx = regions(PRE ? max(w, 2 * a.cw) : w, 128);
  const int nsy = regions(PRE ? max(h, 2 * a.ch) : h, RY);
  const int sx = region % nsx, sy = region / nsx;
  const int x0 = (128 - 2 * kHalo) * sx, y0 = (RY - 2 * kHalo) * sy;
  const int X = x0 + 4 * lane, y = y0 + R * wid;  // the lane's first column and row
  const bool ext = EXT && a.ext != 0, zg = a.zgbc != 0;
  const bool first = sx == 0, has_east = w - 1 - x0 < 128;
  // stored columns and rows
  const bool mine = (lane >= 2 || first) && (lane < 30 || sx == nsx - 1);
  const int ya = sy == 0 ? 0 : y0 + kHalo, yb = sy == nsy - 1 ? y0 + RY : y0 + RY - kHalo;
  // a row's f (16 or 8 bytes per lane), then its factors: pairs (0, 2), (1, 3)
  unsigned char *const rowm = smem + M::fac + R * wid * 1024;
  auto frow = [&](int r) { return reinterpret_cast<S *>(rowm + r * 1024) + 4 * lane; };
  auto fac = [&](int r, int pair) -> float2 & {
    return reinterpret_cast<float2 *>(rowm + r * 1024 + 512)[32 * pair + lane];
  };
  float2 *const xch = reinterpret_cast<float2 *>(smem + M::xch) + lane;
  float2 *const res = reinterpret_cast<float2 *>(smem + M::res) + lane;
  const float2 *const lut = reinterpret_cast<const float2 *>(smem + M::lut);
  const float *const factor = reinterpret_cast<const float *>(lut);
  // exchanged rows: buffer (half sweep parity), warp, its first or last row
  auto slot = [&](int buf, int wd, int lastrow) -> float2 & {
    return xch[((buf * (NW + 2) + 1 + wd) * 2 + lastrow) * 32];
  };

  // ---- loads: all in flight together; f is copied to shared memory (16
  // registers less while the rest arrives, and there for the residual)
  const bool inner = !first && !has_east && y0 > 0 && y0 + RY < h - 1;  // no bounds to check
  griddep_wait();
  const bool colok = X < w;
  const size_t o0 = (size_t)y * P + X;
  float4 pv[R];
  unsigned cw[R];
  unsigned inmask = ~0u;  // columns that are smoothed
  if (inner) {
#pragma unroll
    for (int r = 0; r < R; r++) copy_async<4 * (int)sizeof(S)>(frow(r), a.rhs + o0 + r * P, true);
    if (!a.zero_init) {
#pragma unroll
      for (int r = 0; r < R; r++) pv[r] = St::ldg4(a.in + o0 + r * P);
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) pv[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < R; r++)
      cw[r] = __ldg(reinterpret_cast<const unsigned *>(a.code + o0 + r * P));
  } else {
    unsigned colmask = 0u;
    inmask = 0u;
#pragma unroll
    for (int b = 0; b < 4; b++) {
      colmask |= X + b < w ? 0xffu << (8 * b) : 0u;
      inmask |= X + b >= 1 && X + b < w - 1 ? 0xffu << (8 * b) : 0u;
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const bool ok = colok && y + r < h;
      copy_async<4 * (int)sizeof(S)>(frow(r), a.rhs + (ok ? o0 + r * P : 0), ok);
      pv[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      cw[r] = 0u;
      if (ok) {
        if (!a.zero_init) pv[r] = St::ldg4(a.in + o0 + r * P);
        cw[r] = __ldg(reinterpret_cast<const unsigned *>(a.code + o0 + r * P)) & colmask;
      }
    }
  }
  copy_commit();
  // the coarse level's values and flags under these rows
  constexpr int RC = PRE ? 1 : R / 2 + 1;
  float2 ev[RC];
  unsigned fl[RC];
  if constexpr (!PRE) {
    const int c0 = X >> 1, cy = y >> 1;
#pragma unroll
    for (int k = 0; k < RC; k++) {
      const size_t o = (size_t)(cy + k) * a.cpitch + c0;
      ev[k] = make_float2(0.f, 0.f);
      fl[k] = 0u;
      if (inner || (c0 < a.cw && cy + k < a.ch)) {
        ev[k] = Sc::ldg2(a.ec + o);
        fl[k] = __ldg(reinterpret_cast<const unsigned short *>(a.codec + o)) & 0x0101u;
        if (!inner && c0 + 1 >= a.cw) {
          ev[k].y = 0.0f;
          fl[k] &= 0x00ffu;
        }
      }
    }
  }
  unsigned all = cw[0];
#pragma unroll
  for (int r = 1; r < R; r++) all &= cw[r];
  // the warp's rows or columns touch the domain's edge (rows 1 and h-2 too:
  // their neighbours on the edge follow them); where the edge cells are 0 and
  // stay so, the factor 0 does it
  const bool rim = first || has_east || y <= 1 || y + R >= h - 1;
  const bool wedge = rim && !a.zero_edges;
  const bool west = first && lane == 0;  // column 0 is the lane's first
  const int pe = w - 1 - X;              // place of column w-1 in the lane
  const bool full = __all_sync(0xffffffffu, all == kFull) && !rim;

  if constexpr (!PRE) {
    // ---- prolongate (pressure_solver.cpp:134-172) + correct: an even row
    // lies over one coarse row, an odd row between two
    float ecmul = 1.0f;
    if (EXT && a.scale_bits) coarse_scale(a.scale_bits, a.scale_h1sq, a.scale_kexp, &ecmul);
    float e[3] = {ev[0].x, ev[0].y, __shfl_down_sync(0xffffffffu, ev[0].x, 1)};
    unsigned g = fl[0] | ((__shfl_down_sync(0xffffffffu, fl[0], 1) & 1u) << 16);
#pragma unroll
    for (int k = 0; k < R / 2; k++) {
      const float f[3] = {ev[k + 1].x, ev[k + 1].y, __shfl_down_sync(0xffffffffu, ev[k + 1].x, 1)};
      const unsigned g1 = fl[k + 1] | ((__shfl_down_sync(0xffffffffu, fl[k + 1], 1) & 1u) << 16);
      float u[2][4];
      prolongate2(e, f, g, g1, lut, u);
      if (rim && !ext) {  // no coarse cell beyond: columns and rows from w-2, h-2 on
#pragma unroll
        for (int b = 0; b < 4; b++) {
          if ((b & 1) && X + b >= w - 2) u[0][b] = u[1][b] = 0.0f;
          if (y + 2 * k + 1 >= h - 2) u[1][b] = 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int r = 2 * k + i;
        float *p = &pv[r].x;
        if (EXT && a.scale_bits) {
#pragma unroll
          for (int b = 0; b < 4; b++) u[i][b] = u[i][b] * ecmul;
        }
        if (full) {
#pragma unroll
          for (int b = 0; b < 4; b++) p[b] = rnd<S>(p[b] + u[i][b]);
        } else {
          const unsigned c = y + r >= 1 && y + r < h - 1 ? cw[r] & inmask : 0u;
#pragma unroll
          for (int b = 0; b < 4; b++)
            p[b] = (c >> (8 * b)) & C_CENTER ? rnd<S>(p[b] + u[i][b]) : p[b];
        }
      }
#pragma unroll
      for (int i = 0; i < 3; i++) e[i] = f[i];
      g = g1;
    }
  }

  // ---- registers: pairs of p (0 in solid cells) and of f h^2; factors, with
  // two rows in registers too
  constexpr bool KEEP = R == 2;
  float2 A[R], B[R], FA[R], FB[R], sA[KEEP ? R : 1], sB[KEEP ? R : 1], cA[KEEP ? R : 1],
      cB[KEEP ? R : 1];
  const float hh = a.hh;
  copy_wait();
  float2 sq = make_float2(0.f, 0.f);  // sums of squares of p and (weighted) f h^2
#pragma unroll
  for (int r = 0; r < R; r++) {
    float *p = &pv[r].x;
    const float4 fv = St::lds4(frow(r));
    float F[4] = {fv.x * hh * hh, fv.y * hh * hh, fv.z * hh * hh, fv.w * hh * hh};
    if (!full) {
      const bool brow = y + r == 0 || y + r == h - 1;
      const unsigned in = brow ? 0u : inmask;
      // codes; 32 + flag on the domain's edge (32 where it is and stays 0)
      const unsigned c = (cw[r] & in & 0x1f1f1f1fu) |
                         (~in & (a.zero_edges ? 0x20202020u : (cw[r] & 0x01010101u) | 0x20202020u));
#pragma unroll
      for (int b = 0; b < 4; b++)
        if (!((c >> (8 * b)) & C_CENTER)) p[b] = F[b] = 0.0f;
      float s[4];
#pragma unroll
      for (int b = 0; b < 4; b++) s[b] = factor[(c >> (8 * b)) & 0x3fu];
      if constexpr (KEEP) {
        sA[r] = make_float2(s[0], s[2]);
        sB[r] = make_float2(s[1], s[3]);
        cA[r] = third2(sA[r]);
        cB[r] = third2(sB[r]);
      } else {
        fac(r, 0) = make_float2(s[0], s[2]);
        fac(r, 1) = make_float2(s[1], s[3]);
      }
    }
    A[r] = make_float2(p[0], p[2]);
    B[r] = make_float2(p[1], p[3]);
    FA[r] = make_float2(F[0], F[2]);
    FB[r] = make_float2(F[1], F[3]);
    const float2 ga = kIsHalf<S> ? f2_mul(FA[r], f2(kWeightF<S>)) : FA[r],
                 gb = kIsHalf<S> ? f2_mul(FB[r], f2(kWeightF<S>)) : FB[r];
    sq = f2_fma(gb, gb, f2_fma(ga, ga, f2_fma(B[r], B[r], f2_fma(A[r], A[r], sq))));
  }
  if (!PRE && wedge && zg) {  // edge cells: their inner neighbours' values
    auto flag = [&](unsigned c, int b, float v) { return (c >> (8 * b)) & C_CENTER ? v : 0.0f; };
#pragma unroll
    for (int r = 0; r < R; r++) {
      const float left = __shfl_up_sync(0xffffffffu, B[r].y, 1);
      const unsigned c = cw[r];
      if (west) A[r].x = flag(c, 0, B[r].x);
      if (pe == 0) A[r].x = flag(c, 0, left);
      if (pe == 1) B[r].x = flag(c, 1, A[r].x);
      if (pe == 2) A[r].y = flag(c, 2, B[r].x);
      if (pe == 3) B[r].y = flag(c, 3, A[r].y);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const unsigned c = cw[r];
      if ((r == 0 && y == 0) || (r > 0 && y + r == h - 1)) {
        const int i = r == 0 ? 1 : r - 1;
        A[r] = make_float2(flag(c, 0, A[i].x), flag(c, 2, A[i].y));
        B[r] = make_float2(flag(c, 1, B[i].x), flag(c, 3, B[i].y));
      }
    }
  }
  // (row h-1 as a warp's first row is written by the warp below it)
  if (!(!PRE && wedge && zg && wid > 0 && y == h - 1)) slot(0, wid, 0) = A[0];
  if (!PRE && wedge && zg && wid < NW - 1 && y + R == h - 1)
    slot(0, wid + 1, 0) = make_float2((cw[R - 1] & C_N) ? A[R - 1].x : 0.0f,
                                      ((cw[R - 1] >> 16) & C_N) ? A[R - 1].y : 0.0f);
  slot(0, wid, 1) = B[R - 1];
  if (wid == 0)
    slot(0, -1, 1) = slot(1, -1, 1) = slot(0, NW, 0) = slot(1, NW, 0) = res[0] =
        make_float2(0.f, 0.f);
  // false for infinities and NaNs too
  const bool careful = __syncthreads_or(!(sq.x + sq.y < kBigSq<S>)) != 0;
  // the block's barrier from any of the variants below
  auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); };

  // ---- three sweeps.  Red updates the pair (1, 3) of even rows and (0, 2)
  // of odd rows, black the others; what a warp reads of its neighbours' rows
  // was updated in the half sweep before.
  // A cell on the domain's edge (factor -1, -0 if solid) takes its inner
  // neighbour's value when its colour is updated (follow), which is then that
  // neighbour's value of the sweep before until the neighbour itself is
  // updated, as the reference's zero-gradient copy between sweeps gives it; or
  // it keeps its own.
  // MODE 0: an all-fluid warp, 1: any flags, 2: and the domain's edge, 3: and
  // sums that may not be finite.
  auto half = [&](auto modec, auto redc, const bool follow) {
    constexpr int MODE = decltype(modec)::value;
    constexpr int RED = decltype(redc)::value;
    constexpr bool EDGE = MODE >= 2;
    const int buf = RED ? 0 : 1;
    const float2 below = slot(buf, wid - 1, 1), above = slot(buf, wid + 1, 0);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const bool onB = ((r & 1) ^ RED) != 0;  // which pair of this row
      float2 &own = onB ? B[r] : A[r];
      float2 W, E;
      if (onB) {
        W = A[r];
        E = make_float2(A[r].y, __shfl_down_sync(0xffffffffu, A[r].x, 1));
      } else {
        W = make_float2(__shfl_up_sync(0xffffffffu, B[r].y, 1), B[r].x);
        E = B[r];
      }
      const float2 Sv = r > 0 ? (onB ? B[r > 0 ? r - 1 : 0] : A[r > 0 ? r - 1 : 0]) : below;
      const float2 Nv = r < R - 1 ? (onB ? B[r < R - 1 ? r + 1 : 0] : A[r < R - 1 ? r + 1 : 0]) : above;
      // (W + E needs no pair of its own: scalar additions, without moves)
      const float2 we = make_float2(W.x + E.x, W.y + E.y);
      float2 v = add2(add2(add2(we, Sv), Nv), onB ? FB[r] : FA[r]);
      float2 n;
      if (MODE == 0) {
        n = make_float2(v.x * 0.25f, v.y * 0.25f);
      } else {
        float2 s, c;
        if constexpr (KEEP) {
          s = onB ? sB[r] : sA[r];
          c = onB ? cB[r] : cA[r];
        } else {
          s = fac(r, onB ? 1 : 0);
          c = third2(s);
        }
        if (EDGE) {
          float2 t = make_float2(!onB && west ? E.x : W.x, W.y);
          if (r == 0 && y == 0) t = Nv;
          if (y + r == h - 1) t = Sv;
          if (!follow) t = own;
          if (__float_as_int(s.x) < 0) v.x = -t.x;
          if (__float_as_int(s.y) < 0) v.y = -t.y;
        }
        if (MODE == 3)
          n = make_float2(scaled_any(v.x, s.x), scaled_any(v.y, s.y));
        else
          n = scaled2(v, s, c);
      }
      n = rnd2<S>(n);
      own = n;
    }
    slot(buf ^ 1, wid, 0) = RED ? B[0] : A[0];
    slot(buf ^ 1, wid, 1) = RED ? A[R - 1] : B[R - 1];
    sync();
  };
  auto sweeps = [&](auto modec) {
    const std::integral_constant<int, 1> red{};
    const std::integral_constant<int, 0> black{};
#pragma unroll 1
    for (int s = 0; s < 3; s++) {
      half(modec, red, zg && (!PRE || s > 0));
      half(modec, black, zg);
    }
  };
  if (full)
    sweeps(std::integral_constant<int, 0>{});
  else if (careful)
    sweeps(std::integral_constant<int, 3>{});
  else if (wedge && (first || has_east || y == 0 || y + R >= h))
    sweeps(std::integral_constant<int, 2>{});
  else
    sweeps(std::integral_constant<int, 1>{});

  griddep_launch();
  // ---- store (ya and yb are multiples of R: all of a warp's rows or none)
  if (inner) {
    if (mine && y >= ya && y < yb) {
#pragma unroll
      for (int r = 0; r < R; r++)
        St::st4(a.out + o0 + r * P, make_float4(A[r].x, B[r].x, A[r].y, B[r].y));
    }
  } else if (!wedge) {
#pragma unroll
    for (int r = 0; r < R; r++)
      if (mine && y + r >= ya && y + r < yb && y + r < h && X < w) {
        S *dst = a.out + (size_t)(y + r) * P + X;
        if (X + 3 < w) {
          St::st4(dst, make_float4(A[r].x, B[r].x, A[r].y, B[r].y));
        } else {
          dst[0] = St::fromf(A[r].x);
          if (X + 1 < w) dst[1] = St::fromf(B[r].x);
          if (X + 2 < w) dst[2] = St::fromf(A[r].y);
        }
      }
  } else {
    // columns 0 and w-1, rows 0 and h-1 (stored with rows 1 and h-2): the
    // inner neighbour's value, or as they were (corners of the reference's
    // hierarchy always)
    auto store = [&](int yy, const float (&o)[4], bool corners) {
      if (!mine || X >= w || yy < ya || yy >= yb) return;
      S *dst = a.out + (size_t)yy * P + X;
      if (X + 3 < w && (corners || !(west || pe == 3))) {
        St::st4(dst, make_float4(o[0], o[1], o[2], o[3]));
      } else {
#pragma unroll
        for (int b = 0; b < 4; b++)
          if (X + b < w && (corners || !((b == 0 && west) || b == pe))) dst[b] = St::fromf(o[b]);
      }
    };
    auto old = [&](int xx, int yy) {
      return a.zero_init ? 0.0f : St::ldg1(a.in + (size_t)yy * P + xx);
    };
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int yy = y + r;
      if (yy >= h) break;
      float o[4] = {A[r].x, B[r].x, A[r].y, B[r].y};
      const float in[4] = {__shfl_up_sync(0xffffffffu, B[r].y, 1), o[0], o[1], o[2]};
      if (zg) {
        if (west) o[0] = o[1];
#pragma unroll
        for (int b = 0; b < 4; b++)
          if (b == pe) o[b] = in[b];
        if (yy >= 1 && yy < h - 1) store(yy, o, true);
        if (yy == 1) store(0, o, ext);
        if (yy == h - 2) store(h - 1, o, ext);
      } else {
#pragma unroll
        for (int b = 0; b < 4; b++)
          if (X + b < w && (yy == 0 || yy == h - 1 || (b == 0 && west) || b == pe))
            o[b] = old(X + b, yy);
        store(yy, o, true);
      }
    }
    // corners that hold what was there before
    if (zg && !ext && a.in != a.out && mine && (west || (pe >= 0 && pe < 4))) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int yy = y + r;
        if ((yy != 0 && yy != h - 1) || yy < ya || yy >= yb) continue;
        S *dst = a.out + (size_t)yy * P;
        if (west) dst[0] = St::fromf(old(0, yy));
        if (pe >= 0 && pe < 4) dst[w - 1] = St::fromf(old(w - 1, yy));
      }
    }
  }

  if constexpr (PRE) {
    // ---- residual (calculateResidualField, pressure_solver.cpp:91-116) of
    // every row, restricted (pressure_solver.cpp:118-132): a lane holds the
    // columns over coarse columns X/2 and X/2 + 1
    // rows below and above: (0, 2) and (1, 3) from the two buffers
    const float2 bA = slot(1, wid - 1, 1), bB = slot(0, wid - 1, 1);
    const float2 tA = slot(0, wid + 1, 0), tB = slot(1, wid + 1, 0);
    float2 tt[R];  // odd rows: 1-2-1 sums; even rows: 2-4-2 sums
#pragma unroll
    for (int r = 0; r < R; r++) {
      const float2 SA = r > 0 ? A[r > 0 ? r - 1 : 0] : bA, SB = r > 0 ? B[r > 0 ? r - 1 : 0] : bB;
      const float2 NA = r < R - 1 ? A[r < R - 1 ? r + 1 : 0] : tA,
                   NB = r < R - 1 ? B[r < R - 1 ? r + 1 : 0] : tB;
      const float l = __shfl_up_sync(0xffffffffu, B[r].y, 1);
      const float rr = __shfl_down_sync(0xffffffffu, A[r].x, 1);
      const float C4[4] = {A[r].x, B[r].x, A[r].y, B[r].y};
      const float4 fv = St::lds4(frow(r));
      const float F4[4] = {fv.x, fv.y, fv.z, fv.w};
      float q[4];
      if (full) {
        const float2 va = add2(add2(make_float2(l + B[r].x, B[r].x + B[r].y), SA), NA);
        const float2 vb = add2(add2(make_float2(A[r].x + A[r].y, A[r].y + rr), SB), NB);
        const float V4[4] = {va.x, vb.x, va.y, vb.y};
        // (-4 c is exact: c is a quarter of a finite sum, or not finite itself;
        // so the fused form is the reference's sum)
#pragma unroll
        for (int b = 0; b < 4; b++)
          q[b] = rnd<S>(F4[b] + __fmaf_rn(-4.0f, C4[b], V4[b]) * a.ihsq);
      } else {
        const unsigned c = y + r >= 1 && y + r < h - 1 ? cw[r] & inmask : 0u;
        float W4[4] = {l, A[r].x, B[r].x, A[r].y}, E4[4] = {B[r].x, A[r].y, B[r].y, rr};
        float S4[4] = {SA.x, SB.x, SA.y, SB.y}, N4[4] = {NA.x, NB.x, NA.y, NB.y};
        if (wedge && zg) {  // the edge cells have this cell's value
#pragma unroll
          for (int b = 0; b < 4; b++) {
            if (X + b == 1) W4[b] = C4[b];
            if (X + b == w - 2) E4[b] = C4[b];
            if (y + r == 1) S4[b] = C4[b];
            if (y + r == h - 2) N4[b] = C4[b];
          }
        }
        residual4(c, C4, W4, E4, S4, N4, F4, a.ihsq, q);
#pragma unroll
        for (int b = 0; b < 4; b++) q[b] = rnd<S>(q[b]);
      }
      const float ql = __shfl_up_sync(0xffffffffu, q[3], 1);
      // 1-2-1 or 2-4-2 (products by powers of two are exact)
      if (r & 1)
        tt[r] = make_float2(__fmaf_rn(q[0], 2.0f, ql) + q[1], __fmaf_rn(q[2], 2.0f, q[1]) + q[3]);
      else
        tt[r] = make_float2(__fmaf_rn(q[1], 2.0f, __fmaf_rn(q[0], 4.0f, ql * 2.0f)),
                            __fmaf_rn(q[3], 2.0f, __fmaf_rn(q[2], 4.0f, q[1] * 2.0f)));
    }
    res[(wid + 1) * 32] = tt[R - 1];
    sync();
    const float2 below = res[wid * 32];
    float rfac = a.rfac;
    if (EXT && a.scale_bits) {
      float inv;
      rfac = rfac * (coarse_scale(a.scale_bits, a.scale_h1sq, a.scale_kexp, &inv) * a.scale_h1sq);
    }
    const int c0 = X >> 1;
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      const int yy = y + r, Y = yy >> 1;
      if (!(mine && y >= ya && y < yb)) continue;
      if (!inner && !(Y < a.ch && c0 < a.cw)) continue;
      const float2 tb = r > 0 ? tt[r > 0 ? r - 1 : 0] : below;
      float v0 = ((tb.x + tt[r].x) + tt[r + 1].x) * rfac;
      float v1 = ((tb.y + tt[r].y) + tt[r + 1].y) * rfac;
      if (rim) {
        const bool yz = Y == 0 || Y == a.ch - 1;
        if (yz || c0 == 0 || c0 >= a.cw - 1) v0 = 0.0f;
        if (yz || c0 + 1 >= a.cw - 1) v1 = 0.0f;
      }
      SC *dst = a.rc + (size_t)Y * a.cpitch + c0;
      if (inner || c0 + 1 < a.cw)
        Sc::sts2(dst, v0, v1);
      else
        dst[0] = Sc::fromf(v0);
    }
  }
}

}  // namespace tile
}  // namespace
}  // namespace ubg
