// Step kernels of the fluid time step: boundary conditions, diffusion,
// semi-Lagrangian bicubic advection, divergence, pressure gradient, and the
// accumulated-velocity update.  Each kernel restates one reference function
// (te42kyfo/ubootgl, file:line in the comments) in the reference's operation
// order; the library is compiled with -fmad=false, so results match the FP32
// CPU restatement bit for bit.
#include "ubg_internal.cuh"

namespace ubg {

thread_local LaunchStats g_stats;
thread_local Profiler *g_prof = nullptr;

const char *kernel_class_name(int kc) {
  static const char *n[KC_COUNT] = {"vbc", "accum", "diffuse", "advect", "divergence", "sinks",
                                    "pbc", "gradient", "cfl", "smooth_l0", "smooth_coarse",
                                    "resid_restrict_l0", "resid_restrict_coarse", "coarsen",
                                    "residual", "tracers", "other", "smooth_l1", "tail", "krylov"};
  return (kc >= 0 && kc < KC_COUNT) ? n[kc] : "?";
}

cudaEvent_t Profiler::next() {
  if (used == pool.size()) {
    cudaEvent_t e;
    cudaEventCreate(&e);
    pool.push_back(e);
  }
  return pool[used++];
}

void Profiler::collect() {
  for (auto &m : marks) {
    float ms = 0.0f;
    if (cudaEventElapsedTime(&ms, pool[m.a], pool[m.b]) == cudaSuccess) {
      total_ms[m.kc] += ms;
      count[m.kc] += 1;
    }
  }
  cudaGetLastError();
  marks.clear();
  used = 0;
}

Profiler::~Profiler() {
  for (auto e : pool) cudaEventDestroy(e);
}

namespace {

constexpr int BX = 32, BY = 8;
constexpr int VX = 64, VY = 4;  // row-vector kernels: 4 faces per thread

__device__ __forceinline__ float ld(const float *p, int pitch, int x, int y) {
  return __ldg(p + (size_t)y * pitch + x);
}
// VBCPar / VBCPer / singlePBC, simulation.cpp:22-78.
__device__ __forceinline__ float vbc_par(int bc, float a, float b) {
  if (bc == UBG_BC_INFLOW) return b;
  if (bc == UBG_BC_OUTFLOW || bc == UBG_BC_OUTFLOW_ZERO_PRESSURE) return a > 0.0f ? a : 0.0f;
  return 0.0f;
}
__device__ __forceinline__ float vbc_per(int bc, float a, float b) {
  if (bc == UBG_BC_INFLOW) return b;
  if (bc == UBG_BC_OUTFLOW || bc == UBG_BC_OUTFLOW_ZERO_PRESSURE) return a > 0.0f ? a : 0.0f;
  return -a;
}
__device__ __forceinline__ float single_pbc(int bc, float a) {
  return bc == UBG_BC_OUTFLOW_ZERO_PRESSURE ? -a : a;
}

// ------------------------------------------------------------------ setVBCs
// The reference first sets the x-edges for every row, then the y-edges for
// every column (which fixes the corners), reading the front buffer and
// writing both buffers.  Phase-1 threads own rows 1..h-2 of the two edge
// columns; phase-2 threads own whole columns of the two edge rows and
// recompute the phase-1 value they need.  The two columns next to each
// corner are handled by the corner's thread, because the corner's phase-1
// value reads the old row-0 value of its neighbour.
template <bool XPAR>
__device__ void vbc_component(const float *s, float *b0, float *b1, int pitch, int w, int h,
                              Bcs bc, int t, float &m) {
  // XPAR: x-edges use VBCPar and y-edges VBCPer (vx); otherwise swapped (vy).
  auto edge_x = [&](int side_bc, float a, float b) {
    return XPAR ? vbc_par(side_bc, a, b) : vbc_per(side_bc, a, b);
  };
  auto edge_y = [&](int side_bc, float a, float b) {
    return XPAR ? vbc_per(side_bc, a, b) : vbc_par(side_bc, a, b);
  };
  auto S = [&](int x, int y) { return s[(size_t)y * pitch + x]; };
  auto put = [&](int x, int y, float v) {
    b0[(size_t)y * pitch + x] = v;
    b1[(size_t)y * pitch + x] = v;
    m = fmaxf(m, fabsf(v));
  };
  auto p1 = [&](int x, int y) {
    if (x == 0) return edge_x(bc.w, S(1, y), S(0, y));
    if (x == w - 1) return edge_x(bc.e, S(w - 2, y), S(w - 1, y));
    return S(x, y);
  };
  int n1 = h - 2;
  if (t < n1) {
    int y = t + 1;
    float l = edge_x(bc.w, S(1, y), S(0, y));
    float r = edge_x(bc.e, S(w - 2, y), S(w - 1, y));
    put(0, y, l);
    put(w - 1, y, r);
    return;
  }
  t -= n1;
  if (t >= w) return;
  int x = t;
  if (x == 1 || x == w - 2) return;  // handled by the corner threads
  float bot = edge_y(bc.s, p1(x, 1), p1(x, 0));
  float top = edge_y(bc.n, p1(x, h - 2), p1(x, h - 1));
  float bot2 = 0.f, top2 = 0.f;
  int x2 = -1;
  if (x == 0) x2 = 1;
  if (x == w - 1) x2 = w - 2;
  if (x2 >= 0) {
    bot2 = edge_y(bc.s, S(x2, 1), S(x2, 0));
    top2 = edge_y(bc.n, S(x2, h - 2), S(x2, h - 1));
  }
  put(x, 0, bot);
  put(x, h - 1, top);
  if (x2 >= 0) {
    put(x2, 0, bot2);
    put(x2, h - 1, top2);
  }
}

// The same boundary values from a thread that knows the value v of interior
// face (x, y): the cells of the edge next to it and, next to two edges, the
// corner.  In the step this replaces six launches of edge cells only (setVBCs
// five times, setPBC), 2 to 3 us each: 107 -> 97 us per step at 256x128.
// old(x, y): the edge's value before, which only an inflow keeps; put(x, y,
// value) stores.  Each edge cell's old value is read by this thread alone, and
// before it is overwritten.
template <bool XPAR, class Old, class Put>
__device__ __forceinline__ void edge_cells(int x, int y, float v, int w, int h, Bcs bc, Old &&old,
                                           Put &&put) {
  auto edge_x = [&](int side, float a, auto &&b) {
    if (side == UBG_BC_INFLOW) return b();
    return XPAR ? vbc_par(side, a, 0.0f) : vbc_per(side, a, 0.0f);
  };
  auto edge_y = [&](int side, float a, auto &&b) {
    if (side == UBG_BC_INFLOW) return b();
    return XPAR ? vbc_per(side, a, 0.0f) : vbc_par(side, a, 0.0f);
  };
  const bool W = x == 1, E = x == w - 2, S = y == 1, N = y == h - 2;
  float l = 0.0f, r = 0.0f;
  if (W) l = edge_x(bc.w, v, [&] { return old(0, y); });
  if (E) r = edge_x(bc.e, v, [&] { return old(w - 1, y); });
#pragma unroll 1
  for (int k = 0; k < 2; k++) {
    if (!(k ? N : S)) continue;
    const int ye = k ? h - 1 : 0, side = k ? bc.n : bc.s;
    if (W)
      put(0, ye, edge_y(side, l, [&] {
            return edge_x(bc.w, old(x, ye), [&] { return old(0, ye); });
          }));
    if (E)
      put(w - 1, ye, edge_y(side, r, [&] {
            return edge_x(bc.e, old(x, ye), [&] { return old(w - 1, ye); });
          }));
    put(x, ye, edge_y(side, v, [&] { return old(x, ye); }));
  }
  if (W) put(0, y, l);
  if (E) put(w - 1, y, r);
}
// Calls fn(x, y) for the faces of a block (4 VX x VY cells) that have an edge
// of vx, vy or p next to them, a face per thread, once the block's faces are
// written (fn reads them back).  As four faces in turn by the thread that wrote
// them, with the old values of every kind of edge read, each of the three
// kernels that do this took 4 us more than without (256x128).
template <class F>
__device__ __forceinline__ void edge_faces(const int bx, const int by, const int W, const int H,
                                           F &&fn) {
  const int x0 = bx * 4 * VX, y0 = by * VY, tid = threadIdx.y * VX + threadIdx.x;
  const bool cols = x0 <= 1 || x0 + 4 * VX > W - 3;
  if (!cols && y0 > 1 && y0 + VY <= H - 3) return;
  __syncthreads();
  // rows 1, H-3 and H-2, then columns 1, W-3 and W-2 of the other rows
#pragma unroll 1
  for (int k = 0; k < 4; k++) {
    int x, y;
    if (k < 3) {
      x = x0 + tid;
      y = k == 0 ? 1 : H - 4 + k;
    } else {
      x = tid / VY == 0 ? 1 : W - 4 + tid / VY;
      y = y0 + tid % VY;
      if (tid >= 3 * VY || x < x0 || x >= x0 + 4 * VX || y <= 1 || y >= H - 3) continue;
    }
    if (y >= y0 && y < y0 + VY && x >= 1 && x <= W - 2) fn(x, y);
  }
}

// Whether faces x .. x + 3 of row y have one next to an edge.
__device__ __forceinline__ bool near_edge(int x, int y, int w, int h) {
  return x <= 1 || x + 3 >= w - 2 || y == 1 || y == h - 2;
}

__device__ __forceinline__ void k_vbc_body(VelBufs v, int fx, int fy, Bcs bc, int do_vx, int do_vy,
                      unsigned int *umax_bits, const int bx, const int by, const int bz) {
  int t = bx * blockDim.x + threadIdx.x;
  int W = v.W, H = v.H;
  int nx = (H - 2) + (W - 1);
  float m = 0.0f;
  if (t < nx) {
    if (do_vx) vbc_component<true>(pick(v.vx, fx), v.vx[0], v.vx[1], v.pitch, W - 1, H, bc, t, m);
  } else if (do_vy) {
    vbc_component<false>(pick(v.vy, fy), v.vy[0], v.vy[1], v.pitch, W, H - 1, bc, t - nx, m);
  }
  // max |boundary value| for the next step's CFL dt (interior faces come
  // from the gradient kernel)
  if (umax_bits) {
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(umax_bits, __float_as_uint(m));
  }
}
__global__ void k_vbc(VelBufs v, int fx, int fy, Bcs bc, int do_vx, int do_vy,
                      unsigned int *umax_bits) {
  griddep_wait();
  k_vbc_body(v, fx, fy, bc, do_vx, do_vy, umax_bits, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ---------------------------------------------- applyAccumulatedVelocity
__global__ void k_accum(float *vx, float *vy, float *ax, float *ay, int pitch, int W, int H) {
  griddep_wait();
  int x = blockIdx.x * BX + threadIdx.x, y = blockIdx.y * BY + threadIdx.y;
  size_t i = (size_t)y * pitch + x;
  if (x >= 1 && x < W - 2 && y >= 1 && y < H - 1) {
    vx[i] = vx[i] + ax[i];
    ax[i] = 0.0f;
  }
  if (x >= 1 && x < W - 1 && y >= 1 && y < H - 2) {
    vy[i] = vy[i] + ay[i];
    ay[i] = 0.0f;
  }
}

// ------------------------------------------------------------- face codes
// vx face (x, y) sits between cells x and x+1; vy face (x, y) between cells
// y and y+1.  Diffusion terms (simulation.cpp:118-126 and 144-152):
//   vx: T1 = vx(x+1,y)*f(x+1,y)*f(x+2,y), T2 = vx(x-1,y)*f(x,y)*f(x-1,y),
//       T3 uses fvn = f(x,y+1)*f(x-1,y+1), T4 uses fvs = f(x,y-1)*f(x-1,y-1)
//   vy: T1 = vy(x,y-1)*f(x,y)*f(x,y-1), T2 = vy(x,y+1)*f(x,y+1)*f(x,y+2),
//       T3 uses fve = f(x+1,y)*f(x+1,y+1), T4 uses fvw = f(x-1,y)*f(x-1,y+1)
// FC_A reproduces the chunked advection loop (simulation.cpp:248-256,
// 300-304): faces from x = 1 in chunks of 8 while the chunk start is below
// width-8, a chunk skipped when none of its lanes passes the fluid test.
__global__ void k_face_codes(const uint8_t *__restrict__ flag, uint8_t *cx, uint8_t *cy, int P,
                             int W, int H) {
  int x = blockIdx.x * BX + threadIdx.x, y = blockIdx.y * BY + threadIdx.y;
  auto F = [&](int xx, int yy) -> unsigned { return flag[(size_t)yy * P + xx]; };
  if (x < W - 1 && y < H) {
    unsigned c = 0;
    if (x >= 1 && x < W - 2 && y >= 1 && y < H - 1) {
      if (F(x, y) & F(x + 1, y)) c |= FC_M;
      if (F(x + 1, y) & F(x + 2, y)) c |= FC_T1;
      if (F(x, y) & F(x - 1, y)) c |= FC_T2;
      if (F(x, y + 1) & F(x - 1, y + 1)) c |= FC_T3;
      if (F(x, y - 1) & F(x - 1, y - 1)) c |= FC_T4;
      int xs = 1 + ((x - 1) >> 3) * 8;
      if (xs < (W - 1) - 8)
        for (int i = 0; i < 8; i++)
          if (F(xs - 1 + i, y) & F(xs + i, y)) {
            c |= FC_A;
            break;
          }
    }
    cx[(size_t)y * P + x] = (uint8_t)c;
  }
  if (x < W && y < H - 1) {
    unsigned c = 0;
    if (x >= 1 && x < W - 1 && y >= 1) {
      // rows 1..H-2: the advection loop also covers vy's last row H-2
      if (F(x, y) & F(x, y + 1)) c |= FC_M;
      if (y < H - 2) {
        if (F(x, y) & F(x, y - 1)) c |= FC_T1;
        if (F(x, y + 1) & F(x, y + 2)) c |= FC_T2;
        if (F(x + 1, y) & F(x + 1, y + 1)) c |= FC_T3;
        if (F(x - 1, y) & F(x - 1, y + 1)) c |= FC_T4;
      }
      int xs = 1 + ((x - 1) >> 3) * 8;
      if (xs < W - 8)
        for (int i = 0; i < 8; i++)
          if (F(xs + i, y) & F(xs + i, y - 1)) {
            c |= FC_A;
            break;
          }
    }
    cy[(size_t)y * P + x] = (uint8_t)c;
  }
}

// ---------------------------------------------------------------- diffuse
// One Jacobi sweep, simulation.cpp:114-128 (vx) and 140-154 (vy).  With
// flags in {0, 1}: v*f*f is f*f ? v : 0, v*fv + (1-fv)*(-c) is fv ? v : -c,
// and the running sum starts at +0, so the face codes give the reference's
// values (a zero's sign aside).
// Row-vector access: a thread handles 4 consecutive faces of one row with
// float4 loads (x is a multiple of 4 and rows are 128-byte aligned); a block
// of 64 x 4 threads covers 256 x 4 faces.
__device__ __forceinline__ float4 ld4(const float *p, int P, int x, int y) {
  return __ldg(reinterpret_cast<const float4 *>(p + (size_t)y * P + x));
}
__device__ __forceinline__ float comp(const float4 &v, int j) {
  return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
}
__device__ __forceinline__ unsigned compu(const uchar4 &v, int j) {
  return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
}
// Stores the faces of [x, x+4) that lie in [lo, hi] (a whole float4 when all do).
__device__ __forceinline__ void st4_masked(float *row, int x, int lo, int hi, const float o[4]) {
  if (x >= lo && x + 3 <= hi) {
    *reinterpret_cast<float4 *>(row + x) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (x + j >= lo && x + j <= hi) row[x + j] = o[j];
  }
}

// Four faces of a sweep: (c + a val) / den where the face is open, 0
// elsewhere, val the sum of the neighbours t1 .. t4 in the reference's order.
// Faces with only open neighbours (codes k) need no selects, and the division
// one range check for the four: the sweep is bound by issue as much as by
// memory (405 -> 316 warp instructions per 8 faces a thread; two sweeps with
// their setVBCs at 4096x2048 83.5 -> 76.8 us.  A sweep moves 151 MB, 22 us at the
// copy rate).
__device__ __forceinline__ void diffuse4(unsigned k, const float (&c)[4], const float (&t1)[4],
                                         const float (&t2)[4], const float (&t3)[4],
                                         const float (&t4)[4], float a, float den, float rden,
                                         float (&o)[4]) {
  constexpr unsigned kOpen = (FC_M | FC_T1 | FC_T2 | FC_T3 | FC_T4) * 0x01010101u;
  const bool open = (k & kOpen) == kOpen;
  float x[4];
  if (open) {
#pragma unroll
    for (int j = 0; j < 4; j++) x[j] = c[j] + a * (((t1[j] + t2[j]) + t3[j]) + t4[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const unsigned q = k >> (8 * j);
      float val = 0.0f;
      val = val + ((q & FC_T1) ? t1[j] : 0.0f);
      val = val + ((q & FC_T2) ? t2[j] : 0.0f);
      val = val + ((q & FC_T3) ? t3[j] : -c[j]);
      val = val + ((q & FC_T4) ? t4[j] : -c[j]);
      x[j] = c[j] + a * val;
    }
  }
  // div_rn, its range checked once for the four (zeros are exact too)
  unsigned lo = ~0u;
  float m = 0.0f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    lo = min(lo, div_key(x[j]));
    m = m + fabsf(x[j]);
  }
  if (lo >= kDivKeyLo && m <= 0x1p+100f) {
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const float2 xx = make_float2(x[j], x[j + 1]);
      const float2 q0 = f2_mul(xx, f2(rden));
      const float2 q = f2_fma(f2_fma(q0, f2(-den), xx), f2(rden), q0);
      o[j] = q.x;
      o[j + 1] = q.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = x[j] / den;
  }
  if (!open) {
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = ((k >> (8 * j)) & FC_M) ? o[j] : 0.0f;
  }
}

// edges: 0 = the sweep alone; 1, 2 = the first / second sweep of a step, with
// setVBCs after it (into the sweep's result) and, for vy before the first
// sweep, the boundary values that setVBCs gives the field as it is.  The
// first sweep's vx edges come from the buffer it writes (setVBCs reads that
// buffer's own edge values), every other from the one it reads.
template <int EDGES>
__device__ __forceinline__ void k_diffuse_body(const VelBufs &v, int srcx, int srcy,
                                               const StepScalars *__restrict__ sc, int comps,
                                               Bcs bc, const int bx, const int by) {
  const int x = 4 * (bx * VX + threadIdx.x), y = by * VY + threadIdx.y;
  const int W = v.W, H = v.H, P = v.pitch;
  const float a = sc->a, den = sc->den, rden = sc->rden;
  if ((comps & 1) && y >= 1 && y < H - 1 && x <= W - 3) {
    // vx: interior faces x in [1, W-3], y in [1, H-2]
    const float *s = pick(v.vx, srcx);
    const float4 C = ld4(s, P, x, y), N = ld4(s, P, x, y + 1), S = ld4(s, P, x, y - 1);
    const unsigned K = __ldg(reinterpret_cast<const unsigned *>(v.cx + (size_t)y * P + x));
    const float L = x >= 1 ? ld(s, P, x - 1, y) : 0.0f;
    const float R = x + 4 < W - 1 ? ld(s, P, x + 4, y) : 0.0f;
    const float c[4] = {C.x, C.y, C.z, C.w}, e[4] = {C.y, C.z, C.w, R}, w[4] = {L, C.x, C.y, C.z};
    const float n[4] = {N.x, N.y, N.z, N.w}, ss[4] = {S.x, S.y, S.z, S.w};
    float o[4];
    diffuse4(K, c, e, w, n, ss, a, den, rden, o);
    st4_masked(pick(v.vx, 1 - srcx) + (size_t)y * P, x, 1, W - 3, o);
  }
  if ((comps & 2) && y >= 1 && y < H - 2 && x <= W - 2) {
    // vy: interior faces x in [1, W-2], y in [1, H-3]
    const float *s = pick(v.vy, srcy);
    const float4 C = ld4(s, P, x, y), N = ld4(s, P, x, y + 1), S = ld4(s, P, x, y - 1);
    const unsigned K = __ldg(reinterpret_cast<const unsigned *>(v.cy + (size_t)y * P + x));
    const float L = x >= 1 ? ld(s, P, x - 1, y) : 0.0f;
    const float R = x + 4 < W ? ld(s, P, x + 4, y) : 0.0f;
    const float c[4] = {C.x, C.y, C.z, C.w};
    float e[4] = {C.y, C.z, C.w, R}, w[4] = {L, C.x, C.y, C.z};
    float n[4] = {N.x, N.y, N.z, N.w}, ss[4] = {S.x, S.y, S.z, S.w};
    if (EDGES == 1 && near_edge(x, y, W, H - 1)) {  // the edges as setVBCs would set them first
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (x + j == 1) w[j] = vbc_per(bc.w, c[j], w[j]);
        if (x + j == W - 2) e[j] = vbc_per(bc.e, c[j], e[j]);
        if (y == 1) ss[j] = vbc_par(bc.s, c[j], ss[j]);
        if (y == H - 3) n[j] = vbc_par(bc.n, c[j], n[j]);
      }
    }
    float o[4];
    diffuse4(K, c, ss, n, e, w, a, den, rden, o);
    st4_masked(pick(v.vy, 1 - srcy) + (size_t)y * P, x, 1, W - 2, o);
  }
  if (!EDGES) return;
  const float *sx = pick(v.vx, srcx), *sy = pick(v.vy, srcy);
  float *dx = pick(v.vx, 1 - srcx), *dy = pick(v.vy, 1 - srcy);
  const float *ex = EDGES == 1 ? dx : sx;
  edge_faces(bx, by, W, H, [&](int fx, int fy) {
    if ((comps & 1) && fx <= W - 3)
      edge_cells<true>(
          fx, fy, dx[(size_t)fy * P + fx], W - 1, H, bc,
          [&](int a, int b) { return ex[(size_t)b * P + a]; },
          [&](int a, int b, float q) { dx[(size_t)b * P + a] = q; });
    if ((comps & 2) && fy <= H - 3)
      edge_cells<false>(
          fx, fy, dy[(size_t)fy * P + fx], W, H - 1, bc,
          [&](int a, int b) { return sy[(size_t)b * P + a]; },
          [&](int a, int b, float q) { dy[(size_t)b * P + a] = q; });
  });
}
// On small grids a block takes one component of the velocity (blockIdx.z), which
// fills the chip sooner: 1440x720 164 us per step against 171 with both one after
// the other, 512x256 86.5 against 88.4.  From 3000 blocks per component on it takes
// both, half as many blocks with twice the work each: two sweeps with their
// setVBCs 40 us against 43 at 2900x1450 (4356 blocks), 234 against 248 at
// 8192x4096 (1838 against 1854 per step); at 2045x1021 (2048 blocks) a step takes
// 221 us either way.  The members of a batch fill the chip as they are and take
// both (16 served simulations: 9.09 against 9.16 ms).
constexpr unsigned kSplitBlocks = 3000;
template <int EDGES>
__global__ void __launch_bounds__(256) k_diffuse(VelBufs v, int srcx, int srcy,
                                                 const StepScalars *__restrict__ sc, int comps,
                                                 Bcs bc) {
  griddep_wait();
  const int c = gridDim.z == 1 ? comps : comps & (1 << blockIdx.z);
  k_diffuse_body<EDGES>(v, srcx, srcy, sc, c, bc, blockIdx.x, blockIdx.y);
  griddep_launch();
}

// ----------------------------------------------------------------- advect
// CubicHermite (interpolators.hpp:78-85) is the Catmull-Rom cubic; it is
// evaluated through its four weights of t (the same polynomial, regrouped),
// wA = t(-1/2 + t(1 - t/2)), wB = 1 + t^2(-5/2 + 3t/2),
// wC = t(1/2 + t(2 - 3t/2)), wD = t^2(-1/2 + t/2), with explicit fused
// multiply-adds, exactly as the CPU restatement does.
struct CrW {
  float a, b, c, d;
};
__device__ __forceinline__ float cr_dot(const CrW &w, float A, float B, float C, float D) {
  return __fmaf_rn(w.d, D, __fmaf_rn(w.c, C, __fmaf_rn(w.b, B, w.a * A)));
}

// Two weight sets at once, lane by lane.
struct CrW2 {
  float2 a, b, c, d;
};
__device__ __forceinline__ CrW2 cr_weights2(float2 t) {
  const float2 t2 = f2_mul(t, t);
  CrW2 w;
  w.a = f2_mul(t, f2_fma(t, f2_fma(f2(-0.5f), t, f2(1.0f)), f2(-0.5f)));
  w.b = f2_fma(t2, f2_fma(f2(1.5f), t, f2(-2.5f)), f2(1.0f));
  w.c = f2_mul(t, f2_fma(t, f2_fma(f2(-1.5f), t, f2(2.0f)), f2(0.5f)));
  w.d = f2_mul(t2, f2_fma(f2(0.5f), t, f2(-0.5f)));
  return w;
}
__device__ __forceinline__ float2 cr_dot2(const CrW2 &w, float2 A, float2 B, float2 C, float2 D) {
  return f2_fma(w.d, D, f2_fma(w.c, C, f2_fma(w.b, B, f2_mul(w.a, A))));
}

// Catmull-Rom sample from 16 values (rows r0..r3 of a 4x4 stencil): the
// four vertical dots cr_dot(wy, column j) two columns per instruction, then
// the horizontal dot.
__device__ __forceinline__ float bicubic16(const float *b, int stride, float sx, float sy) {
  const CrW2 w = cr_weights2(make_float2(sy, sx));
  const float2 wa = f2(w.a.x), wb = f2(w.b.x), wc = f2(w.c.x), wd = f2(w.d.x);
  float2 col[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const float2 A = make_float2(b[2 * j], b[2 * j + 1]);
    const float2 B = make_float2(b[stride + 2 * j], b[stride + 2 * j + 1]);
    const float2 C = make_float2(b[2 * stride + 2 * j], b[2 * stride + 2 * j + 1]);
    const float2 D = make_float2(b[3 * stride + 2 * j], b[3 * stride + 2 * j + 1]);
    col[j] = f2_fma(wd, D, f2_fma(wc, C, f2_fma(wb, B, f2_mul(wa, A))));
  }
  const CrW wx{w.a.y, w.b.y, w.c.y, w.d.y};
  return cr_dot(wx, col[0].x, col[0].y, col[1].x, col[1].y);
}

// Shared memory by 32-bit address (kept in a register over a loop, where a
// pointer's window base would be formed again for each access).
__device__ __forceinline__ float lds(unsigned a) {
  float f;
  asm("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(a));
  return f;
}
__device__ __forceinline__ unsigned lds8(unsigned a) {
  unsigned r;
  asm("ld.shared.u8 %0, [%1];" : "=r"(r) : "r"(a));
  return r;
}

// A staged window of one staggered component: region [sx0, sx0+SW) x
// [sy0, sy0+SH) of the grid in shared memory.
struct Win {
  const float *s;
  int sx0, sy0;
};

// bicubicSample (interpolators.hpp:92-206) with the stencil in global memory.
__device__ __noinline__ float bicubic_global(const float *__restrict__ g, int P, float hx, float hy,
                                             float cx, float cy) {
  cx = fmaxf(fminf(cx, hx), 3.0f);
  cy = fmaxf(fminf(cy, hy), 3.0f);
  const int ix = (int)cx, iy = (int)cy;
  return bicubic16(g + (size_t)(iy - 1) * P + (ix - 1), P, cx - (float)ix, cy - (float)iy);
}

// Two bicubic samples at once, lane x of vx at (cx.x, cy.x) and lane y of vy
// at (cx.y, cy.y), the stencils from the shared-memory windows when both lie
// inside, else from global memory.  The coordinates are clamped to [3, h] as
// the reference clamps them (fminf and fmaxf give a NaN the same bounds), so
// c + 2^23 rounded down holds the integer part in its low bits, for grids of
// up to 2^23 cells a side; for wider ones the caller's offsets ox, oy (2^23's
// bits and the window's corner) leave every stencil outside.
struct Pair {
  const float *sx, *sy, *gx, *gy;
  float hxx, hxy, hyx, hyy;  // upper bounds: of vx's grid in x, y, of vy's
  unsigned ox, oy;
  int P;
};
template <int SW, int SH, int SS>
__device__ __forceinline__ float2 bicubic_pair(const Pair &q, float2 cx, float2 cy) {
  const float2 x = make_float2(fmaxf(fminf(cx.x, q.hxx), 3.0f), fmaxf(fminf(cx.y, q.hyx), 3.0f));
  const float2 y = make_float2(fmaxf(fminf(cy.x, q.hxy), 3.0f), fmaxf(fminf(cy.y, q.hyy), 3.0f));
  const float2 tx = f2_add_rm(x, f2(0x1p23f)), ty = f2_add_rm(y, f2(0x1p23f));
  const unsigned ax = __float_as_uint(tx.x) - q.ox, bx = __float_as_uint(tx.y) - q.ox;
  const unsigned ay = __float_as_uint(ty.x) - q.oy, by = __float_as_uint(ty.y) - q.oy;
  if (max(ax, bx) <= SW - 4 && max(ay, by) <= SH - 4) {
    const CrW2 wx = cr_weights2(f2_fma(f2_add_rm(tx, f2(-0x1p23f)), f2(-1.0f), x));
    const CrW2 wy = cr_weights2(f2_fma(f2_add_rm(ty, f2(-0x1p23f)), f2(-1.0f), y));
    const float *a = q.sx + (ay * SS + ax), *b = q.sy + (by * SS + bx);
    float2 col[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
      col[j] = cr_dot2(wy, make_float2(a[j], b[j]), make_float2(a[SS + j], b[SS + j]),
                       make_float2(a[2 * SS + j], b[2 * SS + j]),
                       make_float2(a[3 * SS + j], b[3 * SS + j]));
    return cr_dot2(wx, col[0], col[1], col[2], col[3]);
  }
  return make_float2(bicubic_global(q.gx, q.P, q.hxx, q.hxy, cx.x, cy.x),
                     bicubic_global(q.gy, q.P, q.hyx, q.hyy, cx.y, cy.y));
}

// The same where every stencil lies in the windows, in two parts: the stencils'
// places and weights, and the values; addresses are 32-bit ones of shared
// memory, with 2^23's bits and the window's corner taken off the bases.
template <int SS, int DY>  // vy's window is DY bytes after vx's
struct Near {
  float hxx, hxy, hyx, hyy;
  unsigned base;
  struct At {
    CrW2 wx, wy;
    unsigned a, b;
  };
  // CLAMP: false where no trace of the block reaches the domain's edge
  template <bool CLAMP>
  __device__ __forceinline__ At at(float2 x, float2 y) const {
    if (CLAMP) {
      x = make_float2(fmaxf(fminf(x.x, hxx), 3.0f), fmaxf(fminf(x.y, hyx), 3.0f));
      y = make_float2(fmaxf(fminf(y.x, hxy), 3.0f), fmaxf(fminf(y.y, hyy), 3.0f));
    }
    const float2 tx = f2_add_rm(x, f2(0x1p23f)), ty = f2_add_rm(y, f2(0x1p23f));
    At r;
    r.wx = cr_weights2(f2_fma(f2_add_rm(tx, f2(-0x1p23f)), f2(-1.0f), x));
    r.wy = cr_weights2(f2_fma(f2_add_rm(ty, f2(-0x1p23f)), f2(-1.0f), y));
    r.a = base + 4u * (__float_as_uint(ty.x) * SS + __float_as_uint(tx.x));
    r.b = base + 4u * (__float_as_uint(ty.y) * SS + __float_as_uint(tx.y));
    return r;
  }
  template <int LANE>
  static __device__ __forceinline__ void load(unsigned at, float2 (&v)[16]) {
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const float f = lds(at + 4u * ((k / 4) * SS + k % 4) + (LANE ? DY : 0));
      if (LANE == 0)
        v[k].x = f;
      else
        v[k].y = f;
    }
  }
  static __device__ __forceinline__ float2 value(const At &r, const float2 (&v)[16]) {
    float2 col[4];
#pragma unroll
    for (int j = 0; j < 4; j++) col[j] = cr_dot2(r.wy, v[j], v[4 + j], v[8 + j], v[12 + j]);
    return cr_dot2(r.wx, col[0], col[1], col[2], col[3]);
  }
};

// bilinearSample (interpolators.hpp:11-27) for the advection option: clamp
// to [0, size - 1.1] (glm::clamp = min(max(c, lo), hi)), truncate,
// interpolate along x, then along y; the four values from the shared-memory
// window when they lie inside, else from global memory.
template <int SW, int SH, int SS>
__device__ __forceinline__ float bilinear_win(const Win &wn, const float *__restrict__ g, int P,
                                              int gw, int gh, float cx, float cy) {
  const float hx = (float)gw - 1.1f, hy = (float)gh - 1.1f;
  cx = cx < 0.0f ? 0.0f : cx;
  cx = hx < cx ? hx : cx;
  cy = cy < 0.0f ? 0.0f : cy;
  cy = hy < cy ? hy : cy;
  const int ix = (int)cx, iy = (int)cy;
  const float sx = cx - (float)ix, sy = cy - (float)iy;
  const int lx = ix - wn.sx0, ly = iy - wn.sy0;
  float v1, v2, v3, v4;
  if (lx >= 0 && lx + 1 < SW && ly >= 0 && ly + 1 < SH) {
    const float *b = wn.s + ly * SS + lx;
    v1 = b[0];
    v2 = b[1];
    v3 = b[SS];
    v4 = b[SS + 1];
  } else {
    const float *b = g + (size_t)iy * P + ix;
    v1 = b[0];
    v2 = b[1];
    v3 = b[P];
    v4 = b[P + 1];
  }
  const float vm1 = v1 + (v2 - v1) * sx;
  const float vm2 = v3 + (v4 - v3) * sx;
  return vm1 + (vm2 - vm1) * sy;
}

// advect, simulation.cpp:241-354.  A block handles the vx and vy faces of a
// 64 x TY tile of cells; both velocity components are staged in shared
// memory with a 4-cell halo.
//
// What bounds it: issue (400 warp instructions per 32 cells, of which the
// interpolation is 200) and the FP32 pipe (two operations in each packed
// one), not memory: 124 us at 4096x2048, where 151 MB take 22 us.  It was
// 153 us with each sample by itself.  The steps from there (warp instructions
// per 32 cells, 2048x1024): two samples at once in packed arithmetic, 511; no
// window tests where the staging saw that no value moves far, the end's
// stencil reused from the middle's where it is the same one (mostly: the
// trace bends little in half a step), 492; no clamps away from the domain's
// edge, 441; shared memory by address in a register, 399.  Rows of 96 floats
// instead of 72 took the bank conflicts from 2.0 M to 0.1 M of 8.7 M
// wavefronts.
//
// Tiles of 64 x 4 where 64 x 16 ones would not fill the chip (608 blocks fit
// at once): 256x128 14 -> 6.4 us, 512x256 14 -> 8.5, 1024x512 20.5 -> 17;
// from 2048x1024 on the taller tile stages less (42 against 46 us, 4096x2048
// 124 against 163).  Tiles of 64 x 32 give 47 and 126 us, three blocks per SM
// instead of four 42 and 130.
constexpr int AD_TX = 64, AD_TY = 16, AD_LOW = 4, AD_H = 4;
constexpr unsigned kLowTiles = 608;
// Cells that the fastest value of a window may travel in a step for every
// stencil to lie in it: a sample is at most 1.25^2 times the largest value
// (the sum of the weights' magnitudes), and 1.25^2 * 1.28 = 2 cells plus the
// stencil's own reach stay inside the halo of 4.  (A step at CFL 0.5 moves at
// most half a cell.)
constexpr float kReach = 1.28f;
constexpr int AD_SW = AD_TX + 2 * AD_H;
// Row stride in shared memory: with a multiple of 32, a sample's bank is its
// column, and the lanes of a warp (consecutive faces) read different columns
// whatever rows they fall in.
constexpr int AD_SS = 96;

// BIL: the advection option's bilinearSample instead of bicubicSample.
// EDGES: with the setVBCs that follows in a step, into the buffer written.
template <bool BIL, bool EDGES, int TY>
__device__ __forceinline__ void k_advect_body(const VelBufs &v, int srcx, int srcy,
                                              const StepScalars *__restrict__ sc, Bcs bc,
                                              const int bx, const int by) {
  constexpr int AD_SH = TY + 2 * AD_H;
  // both windows, and both components' codes
  constexpr int kWin = AD_SH * AD_SS, kCodes = TY * AD_TX;
  __shared__ __align__(16) float sv[2 * kWin];
  __shared__ __align__(16) uint8_t codes[2 * kCodes];
  float *const sxv = sv, *const syv = sv + kWin;
  uint8_t *const scx = codes, *const scy = codes + kCodes;
  const int W = v.W, H = v.H, P = v.pitch;
  const float *vx = pick(v.vx, srcx);
  const float *vy = pick(v.vy, srcy);
  const int X0 = bx * AD_TX, Y0 = by * TY;
  const int sx0 = X0 - AD_H, sy0 = Y0 - AD_H;
  const int tid = threadIdx.y * BX + threadIdx.x;
  // staging: 4 entries per load (sx0 and X0 are multiples of 4, so every
  // float4 / uchar4 lies inside its row's pitch); entries outside a
  // component's extent are 0
  const float chalf = sc->chalf, cfull = sc->cfull;
  const bool finite = fabsf(cfull) <= 1e30f && fabsf(chalf) <= fabsf(cfull);
  const float reach = finite ? fminf(kReach / fabsf(cfull), 1e30f) : -1.0f;
  bool far = (W | H) > 1 << 23;
  static_assert(AD_SW % 4 == 0 && AD_H % 4 == 0 && AD_TX % 4 == 0, "vector staging");
  // a warp takes every eighth row, all its loads in flight together
  constexpr int kRows = AD_SH / 8 + (AD_SH % 8 != 0);
  const int lane = threadIdx.x, gx = sx0 + 4 * lane;
  const bool col = lane < AD_SW / 4 && gx >= 0;
  float4 a[kRows], b[kRows];
#pragma unroll
  for (int k = 0; k < kRows; k++) {
    const int ry = threadIdx.y + 8 * k, gy = sy0 + ry;
    a[k] = b[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!col || gy < 0 || (AD_SH % 8 != 0 && ry >= AD_SH)) continue;
    const size_t o = (size_t)gy * P + gx;
    if (gx < W - 1 && gy < H) a[k] = *reinterpret_cast<const float4 *>(vx + o);
    if (gx < W && gy < H - 1) b[k] = *reinterpret_cast<const float4 *>(vy + o);
  }
#pragma unroll
  for (int k = 0; k < kRows; k++) {
    const int ry = threadIdx.y + 8 * k;
    if (gx + 3 >= W - 1) {
      if (gx + 1 >= W - 1) a[k].y = 0.f;
      if (gx + 2 >= W - 1) a[k].z = 0.f;
      a[k].w = 0.f;
      if (gx + 1 >= W) b[k].y = 0.f;
      if (gx + 2 >= W) b[k].z = 0.f;
      if (gx + 3 >= W) b[k].w = 0.f;
    }
    // (each value by itself: a NaN is far)
    far |= !(fabsf(a[k].x) <= reach) | !(fabsf(a[k].y) <= reach) | !(fabsf(a[k].z) <= reach) |
           !(fabsf(a[k].w) <= reach) | !(fabsf(b[k].x) <= reach) | !(fabsf(b[k].y) <= reach) |
           !(fabsf(b[k].z) <= reach) | !(fabsf(b[k].w) <= reach);
    if (lane < AD_SW / 4 && (AD_SH % 8 == 0 || ry < AD_SH)) {
      *reinterpret_cast<float4 *>(sxv + ry * AD_SS + 4 * lane) = a[k];
      *reinterpret_cast<float4 *>(syv + ry * AD_SS + 4 * lane) = b[k];
    }
  }
  for (int i = tid; i < TY * (AD_TX / 4); i += 256) {
    const int ty = i / (AD_TX / 4), tx = 4 * (i - ty * (AD_TX / 4));
    const int x = X0 + tx, y = Y0 + ty;
    unsigned a = 0u, b = 0u;
    if (x < W && y < H) {
      a = __ldg(reinterpret_cast<const unsigned *>(v.cx + (size_t)y * P + x));
      b = __ldg(reinterpret_cast<const unsigned *>(v.cy + (size_t)y * P + x));
    }
    *reinterpret_cast<unsigned *>(scx + ty * AD_TX + tx) = a;
    *reinterpret_cast<unsigned *>(scy + ty * AD_TX + tx) = b;
  }
  // the values of column 0 that the faces of column W - 2 use
  if (X0 + AD_TX > W - 2 && X0 <= W - 2 && tid <= TY)
    far |= !(fabsf(ld(vx, P, 0, min(Y0 + tid, H - 1))) <= reach);
  far = __syncthreads_or(far);
  const Win wx{sxv, sx0, sy0}, wy{syv, sx0, sy0};
  float *outx = pick(v.vx, 1 - srcx), *outy = pick(v.vy, 1 - srcy);
  const bool wide = (W | H) > 1 << 23;
  const Pair q{sxv,
               syv,
               vx,
               vy,
               (float)(W - 1) - 3.0f,
               (float)H - 3.0f,
               (float)W - 3.0f,
               (float)(H - 1) - 3.0f,
               wide ? 0u : 0x4b000000u + (unsigned)(sx0 + 1),
               wide ? 0u : 0x4b000000u + (unsigned)(sy0 + 1),
               P};
  // vx at (cx.x, cy.x), vy at (cx.y, cy.y)
  auto sample = [&](float2 cx, float2 cy) {
    if constexpr (BIL)
      return make_float2(bilinear_win<AD_SW, AD_SH, AD_SS>(wx, vx, P, W - 1, H, cx.x, cy.x),
                         bilinear_win<AD_SW, AD_SH, AD_SS>(wy, vy, P, W, H - 1, cx.y, cy.y));
    else
      return bicubic_pair<AD_SW, AD_SH, AD_SS>(q, cx, cy);
  };
  // (after the barrier: what is read through these is read after it)
  unsigned vbase, cbase;
  asm volatile("mov.u32 %0, %1;" : "=r"(vbase) : "r"((unsigned)__cvta_generic_to_shared(sv)) : "memory");
  asm volatile("mov.u32 %0, %1;" : "=r"(cbase) : "r"((unsigned)__cvta_generic_to_shared(codes)) : "memory");
  const Near<AD_SS, 4 * kWin> near{q.hxx, q.hxy, q.hyx, q.hyy,
                                   vbase - 4u * (q.oy * AD_SS + q.ox)};
  // PATH 0: any trace; 1: every stencil in the windows; 2: and no face or
  // trace of the block near the domain's edge
  auto faces = [&](auto path) {
    constexpr int PATH = decltype(path)::value;
    const int tx = tid % AD_TX, x = X0 + tx;
    const float fx = (float)x;
    float fy = (float)(Y0 + tid / AD_TX);
    int y = Y0 + tid / AD_TX;
    unsigned at0 = vbase + 4u * ((AD_H + tid / AD_TX) * AD_SS + AD_H + tx), ac = cbase + tid;
    // vx and vy in this row and the one below, at this column and the next
    auto px = [&](int dx, int dy) { return lds(at0 + 4u * (dy * AD_SS + dx)); };
    auto py = [&](int dx, int dy) { return lds(at0 + 4u * (kWin + dy * AD_SS + dx)); };
#pragma unroll 1
    for (int n = 0; n < TY * AD_TX / 256; n++, y += 256 / AD_TX, fy += 256 / AD_TX,
             at0 += 4u * (256 / AD_TX) * AD_SS, ac += 256) {
      if (PATH < 2 && (y < 1 || y >= H - 1 || x < 1 || x >= W - 1)) continue;
      const unsigned kx = PATH == 2 || x < W - 2 ? lds8(ac) : 0u, ky = lds8(ac + kCodes);
      if (!((kx | ky) & FC_A)) continue;
      const float vxc = px(0, 0), vxs = px(0, -1), vyc = py(0, 0), vys = py(0, -1);
      // vx face (x, y), simulation.cpp:247-298
      const float pxx = fx + 0.5f, pxy = fy;
      const float vy1 = ((vyc + vys) + (py(1, 0) + py(1, -1))) * 0.25f;
      const float mxx = pxx - vxc * chalf, mxy = pxy - vy1 * chalf;
      // vy face (x, y), simulation.cpp:300-347 (rows 1..H-2 of the vx loop).
      // The reference reads vx at flat index x+1+y*(W-1): for x = W-2 that is
      // element 0 of the next row.
      const float pyx = fx, pyy = fy + 0.5f;
      const bool own = PATH == 2 || x + 1 < W - 1;
      const float a2 = own ? px(1, 0) : ld(vx, P, 0, y + 1);
      const float a3 = own ? px(1, -1) : ld(vx, P, 0, y);
      const float vx1 = ((vxc + vxs) + (a2 + a3)) * 0.25f;
      const float myx = pyx - vx1 * chalf, myy = pyy - vyc * chalf;
      // u: vx at the vx face's middle, vy at the vy face's; w: vx at the vy
      // face's middle, vy at the vx face's; r: the ends of both traces
      const float2 ux = make_float2(mxx - 0.5f, myx), uy = make_float2(mxy, myy - 0.5f);
      const float2 wx = make_float2(myx - 0.5f, mxx), wy = make_float2(myy, mxy - 0.5f);
      float2 r;
      auto end_x = [&](float2 u, float2 w) {
        return make_float2((pxx - u.x * cfull) - 0.5f, pyx - w.x * cfull);
      };
      auto end_y = [&](float2 u, float2 w) {
        return make_float2(pxy - w.y * cfull, (pyy - u.y * cfull) - 0.5f);
      };
      if constexpr (PATH > 0) {
        float2 s[16];
        auto at = near.template at<PATH == 1>(wx, wy);
        near.template load<0>(at.a, s);
        near.template load<1>(at.b, s);
        const float2 w = near.value(at, s);
        at = near.template at<PATH == 1>(ux, uy);
        const unsigned a = at.a, b = at.b;
        near.template load<0>(a, s);
        near.template load<1>(b, s);
        const float2 u = near.value(at, s);
        // the ends mostly lie in the stencils just read
        at = near.template at<PATH == 1>(end_x(u, w), end_y(u, w));
        if (at.a != a) near.template load<0>(at.a, s);
        if (at.b != b) near.template load<1>(at.b, s);
        r = near.value(at, s);
      } else {
        const float2 w = sample(wx, wy), u = sample(ux, uy);
        r = sample(end_x(u, w), end_y(u, w));
      }
      if (kx & FC_A) outx[(size_t)y * P + x] = (kx & FC_M) ? r.x : 0.0f;
      // (row H-2 is vy's northern edge: kept only where setVBCs keeps it)
      if ((ky & FC_A) && (!EDGES || PATH == 2 || y < H - 2 || bc.n == UBG_BC_INFLOW))
        outy[(size_t)y * P + x] = (ky & FC_M) ? r.y : 0.0f;
    }
  };
  if (BIL || far)
    faces(std::integral_constant<int, 0>{});
  else if (X0 > 4 && Y0 >= 8 && X0 + AD_TX + 8 <= W && Y0 + TY + 8 <= H)
    faces(std::integral_constant<int, 2>{});
  else
    faces(std::integral_constant<int, 1>{});
  griddep_launch();
  if (!EDGES) return;
  // setVBCs: the edge cells next to the tile's faces, once those are written
  if (X0 > 1 && X0 + AD_TX <= W - 3 && Y0 > 1 && Y0 + TY <= H - 3) return;
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < AD_TX * TY; i += 256) {
    const int ty = i / AD_TX, x = X0 + i - ty * AD_TX, y = Y0 + ty;
    if (y < 1 || y >= H - 1 || x < 1 || x > W - 2) continue;
    if (x <= W - 3 && (x == 1 || x == W - 3 || y == 1 || y == H - 2))
      edge_cells<true>(
          x, y, outx[(size_t)y * P + x], W - 1, H, bc,
          [&](int xx, int yy) { return vx[(size_t)yy * P + xx]; },
          [&](int xx, int yy, float q) { outx[(size_t)yy * P + xx] = q; });
    if (!(x == 1 || x == W - 2 || y == 1 || y >= H - 3)) continue;
    if (y < H - 2) {
      edge_cells<false>(
          x, y, outy[(size_t)y * P + x], W, H - 1, bc,
          [&](int xx, int yy) { return vy[(size_t)yy * P + xx]; },
          [&](int xx, int yy, float q) {
            // an inflow in the north keeps row H-2, which its own faces write
            if (yy != H - 2 || bc.n != UBG_BC_INFLOW) outy[(size_t)yy * P + xx] = q;
          });
    } else if (bc.n == UBG_BC_INFLOW) {
      const size_t row = (size_t)y * P;
      if (!(scy[i] & FC_A)) outy[row + x] = vy[row + x];
      const float o = outy[row + x];
      if (x == 1) outy[row] = vbc_per(bc.w, o, vy[row]);
      if (x == W - 2) outy[row + W - 1] = vbc_per(bc.e, o, vy[row + W - 1]);
    }
  }
}
// umax_zero: max|u|, zeroed for the step's gradient kernel to accumulate (the
// step's dt has been formed from it); another word where the gradient kernel may
// not follow (the tolerance solver can end in an error).
template <bool BIL, bool EDGES, int TY>
__global__ void __launch_bounds__(256, 4) k_advect(VelBufs v, int srcx, int srcy,
                                                const StepScalars *__restrict__ sc, Bcs bc,
                                                unsigned int *umax_zero) {
  griddep_wait();
  if (EDGES && (blockIdx.x | blockIdx.y | threadIdx.x | threadIdx.y) == 0) *umax_zero = 0u;
  k_advect_body<BIL, EDGES, TY>(v, srcx, srcy, sc, bc, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------- divergence
__device__ __forceinline__ void k_divergence_body(const float *__restrict__ vx,
                                                    const float *__restrict__ vy,
                                                    float *__restrict__ f, int P, int W, int H,
                                                    const StepScalars *__restrict__ sc, const int bx, const int by, const int bz) {
  const int x = 4 * (bx * VX + threadIdx.x), y = by * VY + threadIdx.y;
  if (y < 1 || y >= H - 1 || x > W - 2 || x + 3 < 1) return;
  const float ih = sc->ih;
  float4 U = ld4(vx, P, x, y), V = ld4(vy, P, x, y), Vs = ld4(vy, P, x, y - 1);
  float L = x >= 1 ? ld(vx, P, x - 1, y) : 0.0f;
  float o[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float um = j > 0 ? comp(U, j - 1) : L;
    o[j] = -ih * (comp(U, j) - um + comp(V, j) - comp(Vs, j));
  }
  st4_masked(f + (size_t)y * P, x, 1, W - 2, o);
}
__global__ void __launch_bounds__(256) k_divergence(const float *__restrict__ vx,
                                                    const float *__restrict__ vy,
                                                    float *__restrict__ f, int P, int W, int H,
                                                    const StepScalars *__restrict__ sc) {
  griddep_wait();
  k_divergence_body(vx, vy, f, P, W, H, sc, blockIdx.x, blockIdx.y, blockIdx.z);
  griddep_launch();
}

__global__ void k_sinks(float *f, int P, const SinkCell *cells, int n) {
  griddep_wait();
  // The reference writes the cells in list order; later sinks win.
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (int i = 0; i < n; i++) f[(size_t)cells[i].y * P + cells[i].x] = cells[i].v;
}

// ------------------------------------------------------------------ setPBC
__device__ __forceinline__ void k_pbc_body(float *p, int P, int W, int H, Bcs bc, const int bx, const int by, const int bz) {
  int t = bx * blockDim.x + threadIdx.x;
  auto at = [&](int x, int y) -> float & { return p[(size_t)y * P + x]; };
  if (t < H - 2) {
    int y = t + 1;
    at(0, y) = single_pbc(bc.w, at(1, y));
    at(W - 1, y) = single_pbc(bc.e, at(W - 2, y));
    return;
  }
  t -= H - 2;
  if (t >= W) return;
  int x = t;
  // value of column x in rows 1 and H-2 after the x-edge loop
  float a1, a2;
  if (x == 0) {
    a1 = single_pbc(bc.w, at(1, 1));
    a2 = single_pbc(bc.w, at(1, H - 2));
  } else if (x == W - 1) {
    a1 = single_pbc(bc.e, at(W - 2, 1));
    a2 = single_pbc(bc.e, at(W - 2, H - 2));
  } else {
    a1 = at(x, 1);
    a2 = at(x, H - 2);
  }
  at(x, 0) = single_pbc(bc.s, a1);
  at(x, H - 1) = single_pbc(bc.n, a2);
}
__global__ void k_pbc(float *p, int P, int W, int H, Bcs bc) {
  griddep_wait();
  k_pbc_body(p, P, W, H, bc, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ---------------------------------------------------------------- gradient
// Pressure-gradient update; also folds max(|vx|, |vy|) of every interior
// face (after the update) into *umax_bits for the next step's CFL dt.
// EDGES: with setPBC before it (the update reads no edge cell of p) and with
// the setVBCs that ends a step, into both buffers, its values folded into
// max|u| too.
template <bool EDGES>
__device__ __forceinline__ void k_gradient_body(const VelBufs &v, int fx, int fy, float *p,
                                                const StepScalars *__restrict__ sc,
                                                unsigned int *umax_bits, Bcs bc, const int bx,
                                                const int by) {
  const int x = 4 * (bx * VX + threadIdx.x), y = by * VY + threadIdx.y;
  const int W = v.W, H = v.H, P = v.pitch;
  float m = 0.0f;
  if (y >= 1 && y < H - 1 && x <= W - 2 && x + 3 >= 1) {
    const float ih = sc->ih;
    float *vx = pick(v.vx, fx), *vy = pick(v.vy, fy);
    float4 P0 = *reinterpret_cast<const float4 *>(p + (size_t)y * P + x);
    float4 PN = *reinterpret_cast<const float4 *>(p + (size_t)(y + 1) * P + x);
    float PR = x + 4 < W ? p[(size_t)y * P + x + 4] : 0.0f;
    float4 U = *reinterpret_cast<const float4 *>(vx + (size_t)y * P + x);
    float4 V = *reinterpret_cast<const float4 *>(vy + (size_t)y * P + x);
    uchar4 KX = __ldg(reinterpret_cast<const uchar4 *>(v.cx + (size_t)y * P + x));
    uchar4 KY = __ldg(reinterpret_cast<const uchar4 *>(v.cy + (size_t)y * P + x));
    float ox[4], oy[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float p0 = comp(P0, j), pe = j < 3 ? comp(P0, j + 1) : PR;
      float u = comp(U, j), w = comp(V, j);
      bool inx = x + j >= 1 && x + j <= W - 3;
      bool iny = x + j >= 1 && x + j <= W - 2 && y <= H - 3;
      ox[j] = (inx && (compu(KX, j) & FC_M)) ? u - ih * (pe - p0) : u;
      oy[j] = (iny && (compu(KY, j) & FC_M)) ? w - ih * (comp(PN, j) - p0) : w;
      if (inx) m = fmaxf(m, fabsf(ox[j]));
      if (iny) m = fmaxf(m, fabsf(oy[j]));
    }
    st4_masked(vx + (size_t)y * P, x, 1, W - 3, ox);
    if (y <= H - 3) st4_masked(vy + (size_t)y * P, x, 1, W - 2, oy);
  }
  if (EDGES) {
    float *vx = pick(v.vx, fx), *vy = pick(v.vy, fy);
    float *ox = pick(v.vx, 1 - fx), *oy = pick(v.vy, 1 - fy);
    edge_faces(bx, by, W, H, [&](int xx, int yy) {
      if (xx <= W - 3)
        edge_cells<true>(
            xx, yy, vx[(size_t)yy * P + xx], W - 1, H, bc,
            [&](int a, int b) { return vx[(size_t)b * P + a]; },
            [&](int a, int b, float q) {
              vx[(size_t)b * P + a] = ox[(size_t)b * P + a] = q;
              m = fmaxf(m, fabsf(q));
            });
      if (yy <= H - 3)
        edge_cells<false>(
            xx, yy, vy[(size_t)yy * P + xx], W, H - 1, bc,
            [&](int a, int b) { return vy[(size_t)b * P + a]; },
            [&](int a, int b, float q) {
              vy[(size_t)b * P + a] = oy[(size_t)b * P + a] = q;
              m = fmaxf(m, fabsf(q));
            });
      // setPBC, x edges first (so a corner is two of them)
      const float pc = p[(size_t)yy * P + xx];
      const bool w1 = xx == 1, e1 = xx == W - 2;
      const float l = single_pbc(bc.w, pc), r = single_pbc(bc.e, pc);
      if (w1) p[(size_t)yy * P] = l;
      if (e1) p[(size_t)yy * P + W - 1] = r;
      if (yy == 1 || yy == H - 2) {
        float *row = p + (size_t)(yy == 1 ? 0 : H - 1) * P;
        const int side = yy == 1 ? bc.s : bc.n;
        row[xx] = single_pbc(side, pc);
        if (w1) row[0] = single_pbc(side, l);
        if (e1) row[W - 1] = single_pbc(side, r);
      }
    });
  }
  if (umax_bits) {
    // one atomic per block: per-warp atomics on one address serialise
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float red[VX * VY / 32];
    const int tid = threadIdx.y * VX + threadIdx.x;
    if ((tid & 31) == 0) red[tid >> 5] = m;
    __syncthreads();
    if (tid == 0) {
      for (int i = 1; i < VX * VY / 32; i++) m = fmaxf(m, red[i]);
      atomicMax(umax_bits, __float_as_uint(m));
    }
  }
}
template <bool EDGES>
__global__ void __launch_bounds__(256, 6) k_gradient(VelBufs v, int fx, int fy, float *p,
                                                  const StepScalars *__restrict__ sc,
                                                  unsigned int *umax_bits, Bcs bc) {
  griddep_wait();
  k_gradient_body<EDGES>(v, fx, fy, p, sc, umax_bits, bc, blockIdx.x, blockIdx.y);
  griddep_launch();
}

// ------------------------------------------------------ staged host I/O
// Staged inputs become the front velocity (whole arrays, ghosts included),
// with max|u| over every element folded in as k_umax computes it; and the
// current velocity is snapshotted for an asynchronous download.  Kernels
// rather than 2-D device copies: a pitched cudaMemcpy2D between device
// buffers measured ~0.9 TB/s on GB300.
__global__ void __launch_bounds__(256) k_stage_in(const float *__restrict__ inx,
                                                  const float *__restrict__ iny, float *vx,
                                                  float *vy, int P, int W, int H,
                                                  unsigned int *umax_bits) {
  griddep_wait();
  const int x = 4 * (blockIdx.x * VX + threadIdx.x), y = blockIdx.y * VY + threadIdx.y;
  float m = 0.0f;
  if (x < W && y < H) {
    const size_t i = (size_t)y * P + x;
    const float4 a = *reinterpret_cast<const float4 *>(inx + i);
    const float ax[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (x + j < W - 1) m = fmaxf(m, fabsf(ax[j]));
    st4_masked(vx + (size_t)y * P, x, 0, W - 2, ax);
    if (y < H - 1) {
      const float4 b = *reinterpret_cast<const float4 *>(iny + i);
      const float bx[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (x + j < W) m = fmaxf(m, fabsf(bx[j]));
      st4_masked(vy + (size_t)y * P, x, 0, W - 1, bx);
    }
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float red[VX * VY / 32];
  const int tid = threadIdx.y * VX + threadIdx.x;
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < VX * VY / 32; i++) m = fmaxf(m, red[i]);
    atomicMax(umax_bits, __float_as_uint(m));
  }
}

__global__ void __launch_bounds__(256) k_stage_out(const float *__restrict__ vx,
                                                   const float *__restrict__ vy, float *outx,
                                                   float *outy, int P, int W, int H) {
  griddep_wait();
  const int x = 4 * (blockIdx.x * VX + threadIdx.x), y = blockIdx.y * VY + threadIdx.y;
  if (x >= W || y >= H) return;
  const size_t i = (size_t)y * P + x;
  *reinterpret_cast<float4 *>(outx + i) = *reinterpret_cast<const float4 *>(vx + i);
  if (y < H - 1) *reinterpret_cast<float4 *>(outy + i) = *reinterpret_cast<const float4 *>(vy + i);
}

// --------------------------------------------------------------------- CFL
__global__ void __launch_bounds__(256) k_umax(const float *__restrict__ vx,
                                              const float *__restrict__ vy, int P, int W, int H,
                                              unsigned int *umax_bits) {
  griddep_wait();
  // grid-stride over rows; one atomic per block
  float m = 0.0f;
  for (int y = blockIdx.y * 8 + threadIdx.y; y < H; y += gridDim.y * 8)
    for (int x = blockIdx.x * 32 + threadIdx.x; x < W; x += gridDim.x * 32) {
      if (x < W - 1) m = fmaxf(m, fabsf(ld(vx, P, x, y)));
      if (y < H - 1) m = fmaxf(m, fabsf(ld(vy, P, x, y)));
    }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float red[8];
  if (threadIdx.x == 0) red[threadIdx.y] = m;
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    for (int i = 1; i < 8; i++) m = fmaxf(m, red[i]);
    atomicMax(umax_bits, __float_as_uint(m));
  }
}

__device__ __forceinline__ void k_cfl_scalars_body(const unsigned int *umax_bits, float cfl, float h, float mu,
                              float pwidth, int W, StepScalars *sc, const int bx, const int by, const int bz) {
  float umax = __uint_as_float(*umax_bits);
  umax = umax > 1e-7f ? umax : 1e-7f;
  float dt = cfl * h / umax;
  StepScalars s;
  s.dt = dt;
  s.a = dt * mu * ((float)W - 1.0f) / pwidth;
  s.den = 1.0f + 4.0f * s.a;
  s.rden = __frcp_rn(s.den);
  s.ih = 1.0f / h;
  s.chalf = 0.5f * dt * s.ih;
  s.cfull = dt * s.ih;
  *sc = s;
}
__global__ void k_cfl_scalars(const unsigned int *umax_bits, float cfl, float h, float mu,
                              float pwidth, int W, StepScalars *sc) {
  griddep_wait();
  k_cfl_scalars_body(umax_bits, cfl, h, mu, pwidth, W, sc, blockIdx.x, blockIdx.y, blockIdx.z);
}

inline dim3 grid2(int w, int h, int z = 1) { return dim3((w + BX - 1) / BX, (h + BY - 1) / BY, z); }
inline dim3 grid_vec(int w, int h, int z = 1) {
  return dim3((w + 4 * VX - 1) / (4 * VX), (h + VY - 1) / VY, z);
}


// ---------------------------------------------------- multi-member kernels
__global__ void __launch_bounds__(256) k_diffuse_m(const DiffuseM *__restrict__ A, const int *__restrict__ bs, int n,
            unsigned tag, unsigned *err) {
  griddep_wait();
  if (!table_ok(bs, n, tag, err)) return;
  const int m = member_of(bs, n);
  const DiffuseM a = A[m];
  const int l = (int)blockIdx.x - __ldg(bs + m);
  if (a.edges == 1)
    k_diffuse_body<1>(a.v, a.srcx, a.srcy, a.sc, 3, a.bc, l % a.gx, l / a.gx);
  else
    k_diffuse_body<2>(a.v, a.srcx, a.srcy, a.sc, 3, a.bc, l % a.gx, l / a.gx);
}
__global__ void __launch_bounds__(256, 4) k_advect_m(const AdvectM *__restrict__ A, const int *__restrict__ bs, int n,
           unsigned tag, unsigned *err) {
  griddep_wait();
  if (!table_ok(bs, n, tag, err)) return;
  const int m = member_of(bs, n);
  const AdvectM a = A[m];
  const int l = (int)blockIdx.x - __ldg(bs + m);
  if (l == 0 && (threadIdx.x | threadIdx.y) == 0) *a.umax_zero = 0u;
  // fused members advect bicubically (the bilinear option is not fused)
  k_advect_body<false, true, AD_TY>(a.v, a.srcx, a.srcy, a.sc, a.bc, l % a.gx, l / a.gx);
}
__global__ void __launch_bounds__(256) k_divergence_m(const DivergenceM *__restrict__ A, const int *__restrict__ bs, int n,
               unsigned tag, unsigned *err) {
  griddep_wait();
  if (!table_ok(bs, n, tag, err)) return;
  const int m = member_of(bs, n);
  const DivergenceM a = A[m];
  const int l = (int)blockIdx.x - __ldg(bs + m);
  k_divergence_body(a.vx, a.vy, a.f, a.P, a.W, a.H, a.sc, l % a.gx, l / a.gx, 0);
}
__global__ void __launch_bounds__(256, 5) k_gradient_m(const GradientM *__restrict__ A, const int *__restrict__ bs, int n,
             unsigned tag, unsigned *err) {
  griddep_wait();
  if (!table_ok(bs, n, tag, err)) return;
  const int m = member_of(bs, n);
  const GradientM a = A[m];
  const int l = (int)blockIdx.x - __ldg(bs + m);
  k_gradient_body<true>(a.v, a.fx, a.fy, a.p, a.sc, a.umax, a.bc, l % a.gx, l / a.gx);
}
__global__ void k_cfl_m(const CflM *__restrict__ A, const int *__restrict__ bs, int n, unsigned tag,
                        unsigned *err) {
  griddep_wait();
  if (!table_ok(bs, n, tag, err)) return;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const CflM a = A[m];
  k_cfl_scalars_body(a.umax, a.cfl, a.h, a.mu, a.pwidth, a.W, a.sc, 0, 0, 0);
}
}  // namespace

void launch_face_codes(const VelBufs &v, const uint8_t *flag, uint8_t *cx, uint8_t *cy,
                       cudaStream_t st) {
  k_face_codes<<<grid2(v.W, v.H), dim3(BX, BY), 0, st>>>(flag, cx, cy, v.pitch, v.W, v.H);
  UBG_LAUNCH_CHECK();
}

void launch_vbc(const VelBufs &v, int fx, int fy, Bcs bc, bool do_vx, bool do_vy, cudaStream_t st,
                unsigned int *umax_bits) {
  ProfScope ps_(KC_VBC, st);
  int n = (v.H - 2) + (v.W - 1) + (v.H - 3) + v.W;
  launch_pdl(k_vbc, dim3((n + 255) / 256), dim3(256), 0, st, v, fx, fy, bc, do_vx, do_vy, umax_bits);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_accum(const VelBufs &v, int fx, int fy, float *ax, float *ay, cudaStream_t st) {
  ProfScope ps_(KC_ACCUM, st);
  launch_pdl(k_accum, grid2(v.W, v.H), dim3(BX, BY), 0, st, v.vx[fx], v.vy[fy], ax, ay, v.pitch, v.W, v.H);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_diffuse_sweep(const VelBufs &v, int srcx, int srcy, const StepScalars *sc, int comps,
                          cudaStream_t st, int edges, Bcs bc) {
  ProfScope ps_(KC_DIFFUSE, st);
  auto *k = edges == 0 ? k_diffuse<0> : (edges == 1 ? k_diffuse<1> : k_diffuse<2>);
  dim3 grid = grid_vec(v.W, v.H, 2);
  if (grid.x * grid.y >= kSplitBlocks) grid.z = 1;
  launch_pdl(k, grid, dim3(VX, VY), 0, st, v, srcx, srcy, sc, comps, bc);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_advect(const VelBufs &v, int srcx, int srcy, const StepScalars *sc, cudaStream_t st,
                   bool edges, Bcs bc, unsigned int *umax_zero) {
  ProfScope ps_(KC_ADVECT, st);
  dim3 grid((v.W + AD_TX - 1) / AD_TX, (v.H + AD_TY - 1) / AD_TY);
  auto pick_ty = [&](auto ty) {
    constexpr int T = decltype(ty)::value;
    return v.advect_bilinear ? (edges ? k_advect<true, true, T> : k_advect<true, false, T>)
                             : (edges ? k_advect<false, true, T> : k_advect<false, false, T>);
  };
  auto *k = pick_ty(std::integral_constant<int, AD_TY>{});
  if (grid.x * grid.y < kLowTiles) {
    k = pick_ty(std::integral_constant<int, AD_LOW>{});
    grid.y = (v.H + AD_LOW - 1) / AD_LOW;
  }
  launch_pdl(k, grid, dim3(BX, BY), 0, st, v, srcx, srcy, sc, bc, umax_zero);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_divergence(const VelBufs &v, int fx, int fy, float *f, const StepScalars *sc,
                       cudaStream_t st) {
  ProfScope ps_(KC_DIVERGENCE, st);
  launch_pdl(k_divergence, grid_vec(v.W, v.H), dim3(VX, VY), 0, st, v.vx[fx], v.vy[fy], f,
             v.pitch, v.W, v.H, sc);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_sinks(float *f, int pitch, const SinkCell *cells, int n, cudaStream_t st) {
  if (n <= 0) return;
  ProfScope ps_(KC_SINKS, st);
  k_sinks<<<1, 32, 0, st>>>(f, pitch, cells, n);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_pbc(float *p, int pitch, int W, int H, Bcs bc, cudaStream_t st) {
  ProfScope ps_(KC_PBC, st);
  int n = (H - 2) + W;
  launch_pdl(k_pbc, dim3((n + 255) / 256), dim3(256), 0, st, p, pitch, W, H, bc);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_gradient(const VelBufs &v, int fx, int fy, float *p, const StepScalars *sc,
                     unsigned int *umax_bits, cudaStream_t st, bool edges, Bcs bc) {
  ProfScope ps_(KC_GRADIENT, st);
  launch_pdl(edges ? k_gradient<true> : k_gradient<false>, grid_vec(v.W, v.H), dim3(VX, VY), 0, st,
             v, fx, fy, p, sc, umax_bits, bc);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_stage_in(VelBufs &v, int fx, int fy, const float *inx, const float *iny,
                     unsigned int *umax_bits, cudaStream_t st) {
  ProfScope ps_(KC_OTHER, st);
  UBG_CUDA(cudaMemsetAsync(umax_bits, 0, sizeof(unsigned int), st));
  launch_pdl(k_stage_in, grid_vec(v.W, v.H), dim3(VX, VY), 0, st, inx, iny, v.vx[fx], v.vy[fy],
             v.pitch, v.W, v.H, umax_bits);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_stage_out(const VelBufs &v, int fx, int fy, float *outx, float *outy, cudaStream_t st) {
  ProfScope ps_(KC_OTHER, st);
  launch_pdl(k_stage_out, grid_vec(v.W, v.H), dim3(VX, VY), 0, st, v.vx[fx], v.vy[fy], outx, outy,
             v.pitch, v.W, v.H);
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}

void launch_cfl(const VelBufs &v, int fx, int fy, float cfl, float h, float mu, float pwidth,
                unsigned int *umax_bits, StepScalars *sc, cudaStream_t st, bool umax_ready) {
  ProfScope ps_(KC_CFL, st);
  if (umax_ready) {
    launch_pdl(k_cfl_scalars, dim3(1), dim3(1), 0, st, umax_bits, cfl, h, mu, pwidth, v.W, sc);
    UBG_LAUNCH_CHECK();
    g_stats.launches++;
    return;
  }
  UBG_CUDA(cudaMemsetAsync(umax_bits, 0, sizeof(unsigned int), st));
  dim3 g((v.W + BX - 1) / BX, 64);
  if (g.x > 16) g.x = 16;
  launch_pdl(k_umax, g, dim3(BX, BY), 0, st, v.vx[fx], v.vy[fy], v.pitch, v.W, v.H, umax_bits);
  UBG_LAUNCH_CHECK();
  launch_pdl(k_cfl_scalars, dim3(1), dim3(1), 0, st, umax_bits, cfl, h, mu, pwidth, v.W, sc);
  UBG_LAUNCH_CHECK();
  g_stats.launches += 2;
}

}  // namespace ubg

namespace ubg {
int multi_blocks_diffuse(DiffuseM &a) {
  dim3 g = grid_vec(a.v.W, a.v.H);
  a.gx = (int)g.x;
  return (int)(g.x * g.y);
}
int multi_blocks_advect(AdvectM &a) {
  a.gx = (a.v.W + AD_TX - 1) / AD_TX;
  return a.gx * ((a.v.H + AD_TY - 1) / AD_TY);
}
int multi_blocks_divergence(DivergenceM &a) {
  dim3 g = grid_vec(a.W, a.H);
  a.gx = (int)g.x;
  return (int)(g.x * g.y);
}
int multi_blocks_gradient(GradientM &a) {
  dim3 g = grid_vec(a.v.W, a.v.H);
  a.gx = (int)g.x;
  return (int)(g.x * g.y);
}

void launch_multi_step(int kind, const void *args, const int *bs, int n, int blocks,
                       unsigned tag, unsigned *err, cudaStream_t st) {
  switch (kind) {
    case MK_DIFFUSE:
      launch_pdl(k_diffuse_m, dim3(blocks), dim3(VX, VY), 0, st, (const DiffuseM *)args, bs, n, tag, err);
      break;
    case MK_ADVECT:
      launch_pdl(k_advect_m, dim3(blocks), dim3(BX, BY), 0, st, (const AdvectM *)args, bs, n, tag, err);
      break;
    case MK_DIVERGENCE:
      launch_pdl(k_divergence_m, dim3(blocks), dim3(VX, VY), 0, st, (const DivergenceM *)args, bs,
                 n, tag, err);
      break;
    case MK_GRADIENT:
      launch_pdl(k_gradient_m, dim3(blocks), dim3(VX, VY), 0, st, (const GradientM *)args, bs, n, tag, err);
      break;
    case MK_CFL:
      launch_pdl(k_cfl_m, dim3((n + 127) / 128), dim3(128), 0, st, (const CflM *)args, bs, n, tag,
                 err);
      break;
    default:
      throw ArgError("multi-member launch kind");
  }
  UBG_LAUNCH_CHECK();
  g_stats.launches++;
}
}  // namespace ubg
