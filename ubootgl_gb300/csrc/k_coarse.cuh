// The coarse end of the V-cycle in one block, every level's cells in
// registers while it is worked on (included by k_mg.cu after k_tile.cuh).
//
// Levels of at most 128 x 64 cells: a warp holds R consecutive rows, a lane 4
// columns of them, as in k_tile.cuh, so a half sweep is one barrier, a few
// packed additions per row and an exchange of the warps' edge rows.  Between
// its visits a level's e and right-hand side lie in shared memory (rows of
// 4 * lanes columns).  Edge cells of the reference's coarse levels are 0 and
// never updated; a solid cell and an edge cell have the factor 0.  The
// tolerance hierarchy's edge cells follow their inner neighbour, whose own
// value then stands for them.
//
// What bounds it: latency (barriers between phases of a few dozen
// instructions) and, on the largest level, the issue slots of one SM.  128x64
// and down: 32 us (ncu); the same levels and 256x128 in a 16-block cluster
// took 72 us, levels of up to 2048 cells in one block in shared memory 27 us.
// Code size counts here: one copy of the level's code for both directions
// (two row counts x two directions: 50 us, waiting for instructions).
#pragma once

namespace ubg {
namespace {
namespace coarse {

constexpr int kMaxLevels = 12;
constexpr int kWarps = 32, R = 2;
constexpr int kMaxW = 128, kMaxH = R * kWarps;

struct Level {
  int w, h, lanes;        // lanes = ceil(w / 4)
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
// Shared memory before the levels: arguments (indexed by level, which in the
// parameter space would be a load from memory each time), exchanged rows,
// restriction rows, table.
constexpr int kArgs = 0, kArgsBytes = 1024, kXch = kArgs + kArgsBytes, kRes = kXch + 2 * kWarps * 512, kLut = kRes + kWarps * 256,
              kLevels = (kLut + tile::kLutBytes + 15) / 16 * 16;
inline size_t level_bytes(int w, int h) { return (size_t)((w + 3) / 4) * h * 36; }

// One level's registers in a warp (R rows).
struct Regs {
  float2 A[R], B[R], FA[R], FB[R];   // e and f h^2: columns (0, 2) and (1, 3)
  float2 sA[R], cA[R], sB[R], cB[R];  // factors (tile::scaled2)
  unsigned cw[R];
};

template <bool CAREFUL>
__device__ __forceinline__ void half(Regs &q, const Level &L, unsigned char *smem, const int red,
                                     const bool grad) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float2 *const xch = reinterpret_cast<float2 *>(smem + kXch) + lane;
  auto slot = [&](int buf, int wd, int lastrow) -> float2 & {
    return xch[((buf * kWarps + wd) * 2 + lastrow) * 32];
  };
  const int y = R * wid, xe = L.w - 2 - 4 * lane;
  auto body = [&](auto redc) {
    constexpr int RED = decltype(redc)::value;
    const int buf = RED ? 0 : 1;
    float2 below = make_float2(0.f, 0.f), above = below;
    if (wid > 0) below = slot(buf, wid - 1, 1);
    if (wid < kWarps - 1) above = slot(buf, wid + 1, 0);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const bool onB = ((r & 1) ^ RED) != 0;
      float2 &own = onB ? q.B[r] : q.A[r];
      float2 W, E;
      if (onB) {
        W = q.A[r];
        E = make_float2(q.A[r].y, __shfl_down_sync(0xffffffffu, q.A[r].x, 1));
      } else {
        W = make_float2(__shfl_up_sync(0xffffffffu, q.B[r].y, 1), q.B[r].x);
        E = q.B[r];
      }
      float2 Sv = r > 0 ? (onB ? q.B[r > 0 ? r - 1 : 0] : q.A[r > 0 ? r - 1 : 0]) : below;
      float2 Nv =
          r < R - 1 ? (onB ? q.B[r < R - 1 ? r + 1 : 0] : q.A[r < R - 1 ? r + 1 : 0]) : above;
      if (grad) {
        const unsigned c0 = q.cw[r] >> (onB ? 8 : 0), c1 = c0 >> 16;
        if (onB && lane == 0) W.x = (c0 & C_W) ? own.x : 0.0f;
        if (xe == (onB ? 1 : 0)) E.x = (c0 & C_E) ? own.x : 0.0f;
        if (xe == (onB ? 3 : 2)) E.y = (c1 & C_E) ? own.y : 0.0f;
        if (y + r == 1) Sv = make_float2((c0 & C_S) ? own.x : 0.0f, (c1 & C_S) ? own.y : 0.0f);
        if (y + r == L.h - 2)
          Nv = make_float2((c0 & C_N) ? own.x : 0.0f, (c1 & C_N) ? own.y : 0.0f);
      }
      const float2 v = tile::add2(tile::add2(tile::add2(tile::add2(W, E), Sv), Nv),
                                  onB ? q.FB[r] : q.FA[r]);
      const float2 s = onB ? q.sB[r] : q.sA[r], c = onB ? q.cB[r] : q.cA[r];
      if (CAREFUL)
        own = make_float2(tile::scaled_any(v.x, s.x, c.x), tile::scaled_any(v.y, s.y, c.y));
      else
        own = tile::scaled2(v, s, c);
    }
    slot(buf ^ 1, wid, 0) = RED ? q.B[0] : q.A[0];
    slot(buf ^ 1, wid, 1) = RED ? q.A[R - 1] : q.B[R - 1];
    __syncthreads();
  };
  if (red)
    body(std::integral_constant<int, 1>{});
  else
    body(std::integral_constant<int, 0>{});
}

// One visit of level t: down (e = 0; sweeps, and unless it is the coarsest
// level residual and restriction to level t+1) or up (prolongation and
// correction from level t+1, sweeps).  Ends with the level's e in shared
// memory and a barrier.
template <class S>
__device__ __forceinline__ void visit(const Args<S> &a, const int t, const bool up,
                                      unsigned char *smem) {
  using St = Sto<S>;
  const Level &L = a.L[t];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w = L.w, h = L.h, X = 4 * lane, y = R * wid, stride = 4 * L.lanes;
  const bool ext = a.ext != 0, in = lane < L.lanes;
  float *const e = reinterpret_cast<float *>(smem + L.oe) + X;
  const float *const f = reinterpret_cast<const float *>(smem + L.of) + X;
  const uint8_t *const code = smem + L.oc + X;
  float2 *const xch = reinterpret_cast<float2 *>(smem + kXch) + lane;
  float2 *const res = reinterpret_cast<float2 *>(smem + kRes) + lane;
  const float2 *const lut = reinterpret_cast<const float2 *>(smem + kLut);
  auto slot = [&](int buf, int wd, int lastrow) -> float2 & {
    return xch[((buf * kWarps + wd) * 2 + lastrow) * 32];
  };
  const bool last = t == a.nlev - 1;
  const int ns = last ? (ext ? a.ncoarse : 5) : 3;
  if (y >= h) {  // no rows of this level: only the barriers
    slot(0, wid, 0) = slot(0, wid, 1) = slot(1, wid, 0) = slot(1, wid, 1) = make_float2(0.f, 0.f);
    __syncthreads_or(0);
    for (int i = 0; i < 2 * ns; i++) __syncthreads();
    __syncthreads();
    if (!up && !last) __syncthreads();
    return;
  }
  Regs q;
  unsigned inmask = 0u;
#pragma unroll
  for (int b = 0; b < 4; b++) inmask |= X + b >= 1 && X + b < w - 1 ? 0xffu << (8 * b) : 0u;
  const float hh = L.hh;
  bool ok = true;
  float u[2][4];  // the correction of the two rows
  if (up) {
    // coarse rows y/2 and y/2 + 1
    const Level &C = a.L[t + 1];
    const int cs = 4 * C.lanes, cx = X >> 1, cy = y >> 1;
    const float *ec = reinterpret_cast<const float *>(smem + C.oe) + cy * cs + cx;
    const uint8_t *cc = smem + C.oc + cy * cs + cx;
    float2 v0 = make_float2(0.f, 0.f), v1 = v0;
    unsigned g0 = 0u, g1 = 0u;
    // columns past the coarse width hold 0; the last row of an odd height
    // lies over no coarse row
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
    if (!ext) {  // no coarse cell beyond
#pragma unroll
      for (int b = 0; b < 4; b++) {
        if ((b & 1) && X + b >= w - 2) u[0][b] = u[1][b] = 0.0f;
        if (y + 1 >= h - 2) u[1][b] = 0.0f;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int yy = y + r;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), fv = p;
    unsigned c = 0u;  // smoothed cells' codes, 0 elsewhere
    if (in && yy < h) {
      fv = *reinterpret_cast<const float4 *>(f + yy * stride);
      if (yy >= 1 && yy < h - 1)
        c = *reinterpret_cast<const unsigned *>(code + yy * stride) & inmask;
      if (up) p = *reinterpret_cast<const float4 *>(e + yy * stride);
    }
    float *pp = &p.x;
    float F[4] = {fv.x * hh * hh, fv.y * hh * hh, fv.z * hh * hh, fv.w * hh * hh};
    float2 s[4];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      if (up) pp[b] = pp[b] + u[r][b];
      if (!((c >> (8 * b)) & C_CENTER)) pp[b] = F[b] = 0.0f;
      s[b] = lut[(c >> (8 * b)) & 0x1fu];
    }
    ok = ok && ((fabsf(p.x) + fabsf(p.y)) + (fabsf(p.z) + fabsf(p.w))) +
                       ((fabsf(F[0]) + fabsf(F[1])) + (fabsf(F[2]) + fabsf(F[3]))) <
                   tile::kBig;
    q.A[r] = make_float2(p.x, p.z);
    q.B[r] = make_float2(p.y, p.w);
    q.FA[r] = make_float2(F[0], F[2]);
    q.FB[r] = make_float2(F[1], F[3]);
    q.sA[r] = make_float2(s[0].x, s[2].x);
    q.cA[r] = make_float2(s[0].y, s[2].y);
    q.sB[r] = make_float2(s[1].x, s[3].x);
    q.cB[r] = make_float2(s[1].y, s[3].y);
    q.cw[r] = c;
  }
  slot(0, wid, 0) = q.A[0];
  slot(0, wid, 1) = q.B[R - 1];
  const bool careful = __syncthreads_or(!ok) != 0;

  if (!careful) {
#pragma unroll 1
    for (int s = 0; s < ns; s++) {
      half<false>(q, L, smem, 1, ext && (up || s > 0));
      half<false>(q, L, smem, 0, ext && (up || s > 0));
    }
  } else {
#pragma unroll 1
    for (int s = 0; s < ns; s++) {
      half<true>(q, L, smem, 1, ext && (up || s > 0));
      half<true>(q, L, smem, 0, ext && (up || s > 0));
    }
  }

  // ---- e to shared memory, or the result to the top level's array.  Edge
  // cells: 0, or their inner neighbour's value (corners: the diagonal one's)
  const bool top = t == 0 && (up || last);
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int yy = y + r;
    float o[4] = {q.A[r].x, q.B[r].x, q.A[r].y, q.B[r].y};
    if (ext) {
      const float left = __shfl_up_sync(0xffffffffu, q.B[r].y, 1);
      const float inner[4] = {left, o[0], o[1], o[2]};
      if (lane == 0) o[0] = o[1];
#pragma unroll
      for (int b = 0; b < 4; b++)
        if (X + b == w - 1) o[b] = inner[b];
    }
    auto put = [&](int ye) {
      if (!in || ye >= h) return;
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
        *reinterpret_cast<float4 *>(e + ye * stride) = make_float4(o[0], o[1], o[2], o[3]);
      }
    };
    if (!ext || (yy >= 1 && yy < h - 1)) put(yy);
    if (ext && yy == 1) put(0);
    if (ext && yy == h - 2) put(h - 1);
  }
  if (up || last) {
    __syncthreads();
    return;
  }

  // ---- residual (calculateResidualField, pressure_solver.cpp:91-116) and
  // restriction (pressure_solver.cpp:118-132) to level t+1
  float2 bA = make_float2(0.f, 0.f), bB = bA, tA = bA, tB = bA;
  if (wid > 0) {
    bA = slot(1, wid - 1, 1);
    bB = slot(0, wid - 1, 1);
  }
  if (wid < kWarps - 1) {
    tA = slot(0, wid + 1, 0);
    tB = slot(1, wid + 1, 0);
  }
  float2 tt[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const float2 SA = r > 0 ? q.A[r > 0 ? r - 1 : 0] : bA, SB = r > 0 ? q.B[r > 0 ? r - 1 : 0] : bB;
    const float2 NA = r < R - 1 ? q.A[r < R - 1 ? r + 1 : 0] : tA,
                 NB = r < R - 1 ? q.B[r < R - 1 ? r + 1 : 0] : tB;
    const float l = __shfl_up_sync(0xffffffffu, q.B[r].y, 1);
    const float rr = __shfl_down_sync(0xffffffffu, q.A[r].x, 1);
    float4 fv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in && y + r < h) fv = *reinterpret_cast<const float4 *>(f + (y + r) * stride);
    const float C4[4] = {q.A[r].x, q.B[r].x, q.A[r].y, q.B[r].y};
    const float F4[4] = {fv.x, fv.y, fv.z, fv.w};
    float W4[4] = {l, q.A[r].x, q.B[r].x, q.A[r].y},
          E4[4] = {q.B[r].x, q.A[r].y, q.B[r].y, rr};
    float S4[4] = {SA.x, SB.x, SA.y, SB.y}, N4[4] = {NA.x, NB.x, NA.y, NB.y};
    if (ext) {  // the edge cells have this cell's value
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
    if (r & 1)
      tt[r] = make_float2((dl * 1.0f + d[0] * 2.0f) + d[1] * 1.0f,
                          (d[1] * 1.0f + d[2] * 2.0f) + d[3] * 1.0f);
    else
      tt[r] = make_float2((dl * 2.0f + d[0] * 4.0f) + d[1] * 2.0f,
                          (d[1] * 2.0f + d[2] * 4.0f) + d[3] * 2.0f);
  }
  res[wid * 32] = tt[R - 1];
  __syncthreads();
  float2 below = make_float2(0.f, 0.f);
  if (wid > 0) below = res[(wid - 1) * 32];
  const Level &C = a.L[t + 1];
  const int c0 = X >> 1, cs = 4 * C.lanes;
  float *const fc = reinterpret_cast<float *>(smem + C.of) + c0;
#pragma unroll
  for (int r = 0; r < R; r += 2) {
    const int Y = (y + r) >> 1;
    const float2 tb = r > 0 ? tt[r > 0 ? r - 1 : 0] : below;
    float v0 = ((tb.x + tt[r].x) + tt[r + 1].x) * L.rfac;
    float v1 = ((tb.y + tt[r].y) + tt[r + 1].y) * L.rfac;
    const bool yz = Y == 0 || Y >= C.h - 1;
    if (yz || c0 == 0 || c0 >= C.w - 1) v0 = 0.0f;
    if (yz || c0 + 1 >= C.w - 1) v1 = 0.0f;
    if (Y < C.h && c0 < cs) *reinterpret_cast<float2 *>(fc + Y * cs) = make_float2(v0, v1);
  }
  __syncthreads();
}

template <class S>
__device__ __forceinline__ void run(const Args<S> &args, unsigned char *smem) {
  using St = Sto<S>;
  static_assert(sizeof(Args<S>) <= kArgsBytes && sizeof(Args<S>) % 4 == 0, "arguments");
  if (threadIdx.x < sizeof(Args<S>) / 4)
    reinterpret_cast<unsigned *>(smem + kArgs)[threadIdx.x] =
        reinterpret_cast<const unsigned *>(&args)[threadIdx.x];
  __syncthreads();
  const Args<S> &a = *reinterpret_cast<const Args<S> *>(smem + kArgs);
  // codes of every level, the top level's right-hand side (columns past the
  // width: 0)
  for (int t = 0; t < a.nlev; t++) {
    const Level &L = a.L[t];
    const int lane = threadIdx.x & 31, X = 4 * lane, stride = 4 * L.lanes;
    if (lane >= L.lanes) continue;
    unsigned m = 0u;
#pragma unroll
    for (int b = 0; b < 4; b++) m |= X + b < L.w ? 0xffu << (8 * b) : 0u;
    for (int y = threadIdx.x >> 5; y < L.h; y += kWarps) {
      *reinterpret_cast<unsigned *>(smem + L.oc + y * stride + X) =
          __ldg(reinterpret_cast<const unsigned *>(L.code + (size_t)y * L.code_pitch + X)) & m;
      if (t == 0)
        *reinterpret_cast<float4 *>(smem + L.of + (y * stride + X) * 4) =
            St::ldg4(a.rhs_top + (size_t)y * a.rhs_pitch + X);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int v = 0; v < 2 * a.nlev - 1; v++) {
    const bool up = v >= a.nlev;
    visit<S>(a, up ? 2 * a.nlev - 2 - v : v, up, smem);
  }
}

}  // namespace coarse
}  // namespace
}  // namespace ubg
