// Advection stage: scalForward + scalCorrect + velForward + velCorrect of
// shaders/advect.wgsl:36-103 in one kernel per tile.
//
// The first-order values Th, Yh, Uh, Vh (advect.wgsl:68-76, 36-47) exist only
// in shared memory: each CTA computes them on its tile plus a halo of H cells,
// then applies the MacCormack correction (:78-103, :49-66) to its own cells and
// faces. A forward-trace sample that lands outside the staged halo (at most H
// cells wide) recomputes the first-order value from global memory, so the
// result depends on neither the time step nor the tile. Global traffic per cell: U, V, T, Y
// read (through L1), T2, Y2, U2, V2 written; the 40 bytes/cell of Th/Yh and
// 8 bytes/face of Uh/Vh of the reference schedule never reach HBM.
#include "gas_dev.cuh"
#include "kernels.h"

namespace cfg {

namespace {

// at(i, j): the first-order value from shared memory (RW x RH values from (rx0, ry0) on, the faces' rows ST
// words apart), recomputed from global memory outside the staged region; quad(i, j, ...): the 2x2 block straight from shared memory when all four
// corners are inside the level (no boundary rule applies) and inside the staged region
__device__ __forceinline__ bool staged_block(int i, int j, int nx1, int ny1, int rx0, int ry0, int RW, int RH) {
  return (unsigned)i < (unsigned)nx1 && (unsigned)j < (unsigned)ny1 && (unsigned)(i - rx0) < (unsigned)(RW - 1) &&
         (unsigned)(j - ry0) < (unsigned)(RH - 1);
}
// first-order values outside the staged region, from global memory: out of line, so that the
// corrections' fast path stays compact in the instruction cache
__device__ __forceinline__ VelSampler vel_sampler(const SceneDesc& S) {
  VelSampler vs;
  vs.u = UField{S.U, S.nx, S.ny, S.pu};
  vs.v = VField{S.V, S.nx, S.ny, S.pc};
  vs.dx = S.P.dx;
  vs.rdx = __frcp_rn(S.P.dx);
  return vs;
}
__device__ __noinline__ float th_far(const SceneDesc& S, int i, int j) {
  float ox, oy; vel_sampler(S).trace((float)i + 0.5f, (float)j + 0.5f, S.P.dt, ox, oy);
  return sample(CField{S.T, S.nx, S.ny, S.pc, S.P.Tamb}, ox, oy, 0.5f, 0.5f);
}
__device__ __noinline__ float4 yh_far(const SceneDesc& S, int i, int j) {
  float ox, oy; vel_sampler(S).trace((float)i + 0.5f, (float)j + 0.5f, S.P.dt, ox, oy);
  return sample4(C4Field{S.Y, S.nx, S.ny, S.pc, ambY(S.P)}, ox, oy);
}
__device__ __noinline__ float uh_far(const SceneDesc& S, int i, int j) {
  const VelSampler vs = vel_sampler(S);
  float ox, oy; vs.trace((float)i, (float)j + 0.5f, S.P.dt, ox, oy);
  return sample(vs.u, ox, oy, 0.f, 0.5f);
}
__device__ __noinline__ float vh_far(const SceneDesc& S, int i, int j) {
  const VelSampler vs = vel_sampler(S);
  float ox, oy; vs.trace((float)i + 0.5f, (float)j, S.P.dt, ox, oy);
  return sample(vs.v, ox, oy, 0.5f, 0.f);
}
struct ThLookup {
  const float* sm; int rx0, ry0, RW, RH; const SceneDesc* S; const CField* T;
  __device__ __forceinline__ bool quad(int i, int j, float& A, float& C, float& D, float& E) const {
    if (!staged_block(i, j, T->nx - 1, T->ny - 1, rx0, ry0, RW, RH)) return false;
    const float* q = sm + (j - ry0) * RW + (i - rx0);
    A = q[0]; C = q[1]; D = q[RW]; E = q[RW + 1];
    return true;
  }
  __device__ __forceinline__ float at(int i, int j) const {
    if (i < 0 || i >= T->nx || j >= T->ny) return T->amb;
    j = max(j, 0);
    const int ri = i - rx0, rj = j - ry0;
    if (ri >= 0 && ri < RW && rj >= 0 && rj < RH) return sm[rj * RW + ri];
    return th_far(*S, i, j);
  }
};
struct YhLookup {
  const float4* sm; int rx0, ry0, RW, RH; const SceneDesc* S; const C4Field* Y;
  __device__ __forceinline__ bool quad(int i, int j, float4& A, float4& C, float4& D, float4& E) const {
    if (!staged_block(i, j, Y->nx - 1, Y->ny - 1, rx0, ry0, RW, RH)) return false;
    const float4* q = sm + (j - ry0) * RW + (i - rx0);
    A = q[0]; C = q[1]; D = q[RW]; E = q[RW + 1];
    return true;
  }
  __device__ __forceinline__ float4 at(int i, int j) const {
    if (i < 0 || i >= Y->nx || j >= Y->ny) return Y->amb;
    j = max(j, 0);
    const int ri = i - rx0, rj = j - ry0;
    if (ri >= 0 && ri < RW && rj >= 0 && rj < RH) return sm[rj * RW + ri];
    return yh_far(*S, i, j);
  }
};
struct UhLookup {
  const float* sm; int rx0, ry0, RW, RH, ST; const SceneDesc* S; const VelSampler* vs;
  __device__ __forceinline__ bool quad(int i, int j, float& A, float& C, float& D, float& E) const {
    if (!staged_block(i, j, vs->u.nx, vs->u.ny - 1, rx0, ry0, RW, RH)) return false;
    const float* q = sm + (j - ry0) * ST + (i - rx0);
    A = q[0]; C = q[1]; D = q[ST]; E = q[ST + 1];
    return true;
  }
  __device__ __forceinline__ float at(int i, int j) const {
    const UField& u = vs->u;
    if (i < 0 || i > u.nx || j >= u.ny) return 0.f;
    float sgn = 1.f;
    if (j < 0) { j = 0; sgn = -1.f; }
    const int ri = i - rx0, rj = j - ry0;
    float v;
    if (ri >= 0 && ri < RW && rj >= 0 && rj < RH) v = sm[rj * ST + ri];
    else v = uh_far(*S, i, j);
    return sgn < 0.f ? -v : v;
  }
};
struct VhLookup {
  const float* sm; int rx0, ry0, RW, RH, ST; const SceneDesc* S; const VelSampler* vs;
  __device__ __forceinline__ bool quad(int i, int j, float& A, float& C, float& D, float& E) const {
    if (!staged_block(i, j, vs->v.nx - 1, vs->v.ny, rx0, ry0, RW, RH)) return false;
    const float* q = sm + (j - ry0) * ST + (i - rx0);
    A = q[0]; C = q[1]; D = q[ST]; E = q[ST + 1];
    return true;
  }
  __device__ __forceinline__ float at(int i, int j) const {
    const VField& v = vs->v;
    if (i < 0 || i >= v.nx || j > v.ny) return 0.f;
    j = max(j, 0);
    const int ri = i - rx0, rj = j - ry0;
    if (ri >= 0 && ri < RW && rj >= 0 && rj < RH) return sm[rj * ST + ri];
    return vh_far(*S, i, j);
  }
};

}  // namespace

// The velocity at a trace's own starting point (the first half of the midpoint rule), where the
// bilinear weights are 0 and 1/2: a cell centre averages its two U and its two V faces, a face has its
// own component and the average of four of the other. The same values as VelSampler::vel there (its
// products by a weight of 0 add an exact zero).
__device__ __forceinline__ void vel_cell(const VelSampler& s, int i, int j, float& vx, float& vy) {
  const float* u = s.u.a + j * s.u.pu + i;
  const float* v = s.v.a + j * s.v.pc + i;
  vx = div_by_rcp(mixf(__ldg(u), __ldg(u + 1), 0.5f), s.dx, s.rdx);
  vy = div_by_rcp(mixf(__ldg(v), __ldg(v + s.v.pc), 0.5f), s.dx, s.rdx);
}
__device__ __forceinline__ void vel_uface(const VelSampler& s, int i, int j, float& vx, float& vy) {
  const float* v = s.v.a + j * s.v.pc + i;
  const bool w = i > 0, e = i < s.v.nx;   // still air beside the domain
  const float A = w ? __ldg(v - 1) : 0.f, C = e ? __ldg(v) : 0.f;
  const float D = w ? __ldg(v + s.v.pc - 1) : 0.f, E = e ? __ldg(v + s.v.pc) : 0.f;
  vx = div_by_rcp(__ldg(s.u.a + j * s.u.pu + i), s.dx, s.rdx);
  vy = div_by_rcp(mixf(mixf(A, C, 0.5f), mixf(D, E, 0.5f), 0.5f), s.dx, s.rdx);
}
__device__ __forceinline__ void vel_vface(const VelSampler& s, int i, int j, float& vx, float& vy) {
  const float* u = s.u.a + j * s.u.pu + i;
  const bool n = j < s.u.ny;              // still air above, the no-slip ghost -U(i, 0) below
  const float* us = j > 0 ? u - s.u.pu : u;
  const float D = n ? __ldg(u) : 0.f, E = n ? __ldg(u + 1) : 0.f;
  float A = __ldg(us), C = __ldg(us + 1);
  if (j == 0) { A = -A; C = -C; }
  vx = div_by_rcp(mixf(mixf(A, C, 0.5f), mixf(D, E, 0.5f), 0.5f), s.dx, s.rdx);
  vy = div_by_rcp(__ldg(s.v.a + j * s.v.pc + i), s.dx, s.rdx);
}
// the second half of VelSampler::trace from (gx, gy), whose displacement in half the step is (hx, hy) (its negative
// for the trace forward, with -dt)
__device__ __forceinline__ void trace_from(const VelSampler& s, float gx, float gy, float hx, float hy, float tdt,
                                           float& ox, float& oy) {
  float wx, wy; s.vel(gx - hx, gy - hy, wx, wy);
  ox = s.moved(gx, tdt * wx); oy = s.moved(gy, tdt * wy);
}
// sample and the corners' range at one point
template <class F>
__device__ __forceinline__ float sample_range(const F& f, float gx, float gy, float ox, float oy, float& lo, float& hi) {
  float tx, ty;
  const int i = floor_frac(gx - ox, tx), j = floor_frac(gy - oy, ty);
  float A, C, D, E;
  corners(f, i, j, A, C, D, E);
  lo = fminf(fminf(A, C), fminf(D, E)); hi = fmaxf(fmaxf(A, C), fmaxf(D, E));
  return mixf(mixf(A, C, tx), mixf(D, E, tx), ty);
}
// how many cells beyond [x0, x1] x [y0, y1] the corners of a bilinear sample at (gx - ox, gy - oy) lie
__device__ __forceinline__ int beyond(float gx, float gy, float ox, float oy, int x0, int y0, int x1, int y1) {
  float t;
  const int i = floor_frac(gx - ox, t), j = floor_frac(gy - oy, t);
  return max(max(x0 - i, i + 1 - x1), max(y0 - j, j + 1 - y1));
}

// One thread per cell of the tile, with the U face west and the V face south of it. Before the
// barrier a thread traces its own three points both ways from one starting velocity and keeps its
// first-order values, their limits and the points the correction reads back at in registers; the
// tile's threads then share the halo's first-order values, as many cells wide (1 to H) as the
// corrections of this tile read: displacements under a cell at CFL 0.5, one to three cells in the
// app's plumes at its fixed 2-4 ms steps. Bound by instruction issue and fetch: 12.4 M warp
// instructions at 256x384 before (every trace from the general sampler, twice; the limits gathered
// again; two halo cells everywhere, and beyond them four recomputed traces per sample).
// Now (back to back): 20.1 -> 14.9 us at 256x384, 50 -> 37.7 at 512x768 (CFL 0.5; 0.4 us of each for the bound on
// displacements, with the half step's shared by both directions); 26.7 -> 14.2 at 224x320 and 47 -> 29 at 352x512
// (3 and 2 ms steps).
// Registers for three CTAs of 256 threads per SM (80, no spill in the tile's own path): with 64 and
// four CTAs 256x384 took 16.1 instead of 14.6 us, 512x768 36.8 instead of 37.1.
template <int TX, int TY, int H>
__global__ void __launch_bounds__(TX * TY, TX * TY == 256 ? 3 : 2) k_advect(const SceneDesc* __restrict__ scenes, const Work* __restrict__ work) {
  constexpr int NT = TX * TY;
  constexpr int RW = TX + 2 * H, RH = TY + 2 * H;            // cell region
  constexpr int UW = RW + 1, UH = RH;                          // U-face region
  constexpr int VW = RW, VH = RH + 1;                          // V-face region
  __shared__ float sTh[RH * RW];
  __shared__ float4 sYh[RH * RW];
  __shared__ float sUh[UH * UW];
  __shared__ float sVh[VH * VW];
  __shared__ int s_h;

  const Work w = work[blockIdx.x];
  const SceneDesc& S = scenes[w.scene];
  if (!S.enabled) return;
  const int nx = S.nx, ny = S.ny, pc = S.pc, pu = S.pu;
  const float dt = S.P.dt, hd = 0.5f * dt;
  const int x0 = w.tx * TX, y0 = w.ty * TY;
  const int rx0 = x0 - H, ry0 = y0 - H;

  const VelSampler vs = vel_sampler(S);
  const CField Tf{S.T, nx, ny, pc, S.P.Tamb};
  const C4Field Yf{S.Y, nx, ny, pc, ambY(S.P)};

  // ---- own cell, U face and V face: first-order values (advect.wgsl:36-47, 68-76) and limits at the
  // point traced back from, the point traced forward to
  const int li = threadIdx.x % TX, lj = threadIdx.x / TX, i = x0 + li, j = y0 + lj;
  const bool own = i < nx && j < ny;
  const bool last = x0 + TX >= nx || y0 + TY >= ny;   // the tile also owns faces x = nx or y = ny
  float th = 0.f, tlo = 0.f, thi = 0.f, uh = 0.f, ulo = 0.f, uhi = 0.f, vh = 0.f, vlo = 0.f, vhi = 0.f;
  float4 yh = make_float4(0.f, 0.f, 0.f, 0.f), ylo = yh, yhi = yh;
  float cbx = 0.f, cby = 0.f, ubx = 0.f, uby = 0.f, vbx = 0.f, vby = 0.f;
  int far = last ? 2 : 1;   // halo cells the own sites' corrections need
  if (threadIdx.x == 0) s_h = 1;
  __syncthreads();
  if (own) {
    const float gx = (float)i + 0.5f, gy = (float)j + 0.5f;
    float vx, vy, hx, hy, ox, oy;
    auto half = [&] { hx = vs.bounded(hd * vx); hy = vs.bounded(hd * vy); };
    vel_cell(vs, i, j, vx, vy);
    half();
    trace_from(vs, gx, gy, hx, hy, dt, ox, oy);
    {
      float tx, ty;
      const int ci = floor_frac(ox - 0.5f, tx), cj = floor_frac(oy - 0.5f, ty);
      float A, C, D, E;
      corners(Tf, ci, cj, A, C, D, E);
      tlo = fminf(fminf(A, C), fminf(D, E)); thi = fmaxf(fmaxf(A, C), fmaxf(D, E));
      th = mixf(mixf(A, C, tx), mixf(D, E, tx), ty);
      float4 A4, C4, D4, E4;
      corners(Yf, ci, cj, A4, C4, D4, E4);
      ylo = min4(min4(A4, C4), min4(D4, E4)); yhi = max4(max4(A4, C4), max4(D4, E4));
      yh = mix4(mix4(A4, C4, tx), mix4(D4, E4, tx), ty);
    }
    trace_from(vs, gx, gy, -hx, -hy, -dt, cbx, cby);
    far = max(far, beyond(cbx, cby, 0.5f, 0.5f, x0, y0, x0 + TX - 1, y0 + TY - 1));
    const int r = (lj + H) * RW + li + H;
    sTh[r] = th; sYh[r] = yh;
    // U face
    vel_uface(vs, i, j, vx, vy);
    half();
    trace_from(vs, (float)i, gy, hx, hy, dt, ox, oy);
    uh = sample_range(vs.u, ox, oy, 0.f, 0.5f, ulo, uhi);
    trace_from(vs, (float)i, gy, -hx, -hy, -dt, ubx, uby);
    far = max(far, beyond(ubx, uby, 0.f, 0.5f, x0, y0, x0 + TX, y0 + TY - 1));
    sUh[(lj + H) * UW + li + H] = uh;
    // V face
    vel_vface(vs, i, j, vx, vy);
    half();
    trace_from(vs, gx, (float)j, hx, hy, dt, ox, oy);
    vh = sample_range(vs.v, ox, oy, 0.5f, 0.f, vlo, vhi);
    trace_from(vs, gx, (float)j, -hx, -hy, -dt, vbx, vby);
    far = max(far, beyond(vbx, vby, 0.5f, 0.f, x0, y0, x0 + TX - 1, y0 + TY));
    sVh[(lj + H) * VW + li + H] = vh;
  } else if (i == nx && j < ny) {   // the last faces of a domain that ends inside the tile
    float ox, oy; vs.trace((float)nx, (float)j + 0.5f, dt, ox, oy);
    sUh[(lj + H) * UW + li + H] = sample(vs.u, ox, oy, 0.f, 0.5f);
  } else if (j == ny && i < nx) {
    float ox, oy; vs.trace((float)i + 0.5f, (float)ny, dt, ox, oy);
    sVh[(lj + H) * VW + li + H] = sample(vs.v, ox, oy, 0.5f, 0.f);
  }
  if (far > 1) atomicMax(&s_h, min(far, H));
  __syncthreads();
  // ---- first-order values of the halo: the ring of h cells about the tile (U: h + 1 columns east, V: h + 1
  // rows north), the three fields' rings one after the other
  const int h = s_h;
  const int nC = (TX + 2 * h) * (TY + 2 * h) - NT, nU = (TX + 2 * h + 1) * (TY + 2 * h) - NT,
            nV = (TX + 2 * h) * (TY + 2 * h + 1) - NT;
  for (int e0 = threadIdx.x; e0 < nC + nU + nV; e0 += NT) {
    const int f = e0 < nC ? 0 : e0 < nC + nU ? 1 : 2;   // cells, U faces, V faces
    int e = e0 - (f == 0 ? 0 : f == 1 ? nC : nC + nU), a, b;
    // rows below and above the tile first, then the columns beside it
    const int sr = f == 1 ? h + 1 : h, rw = TX + h + sr, rows = (2 * h + (f == 2 ? 1 : 0)) * rw;
    if (e < rows) {
      b = (int)((unsigned)e / (unsigned)rw); a = e - b * rw - h; b = b < h ? b - h : b - h + TY;
    } else {
      e -= rows;
      b = (int)((unsigned)e / (unsigned)(h + sr)); a = e - b * (h + sr); a = a < h ? a - h : a - h + TX;
    }
    const int ci = x0 + a, cj = y0 + b;
    if (ci < 0 || ci >= nx + (f == 1 ? 1 : 0) || cj < 0 || cj >= ny + (f == 2 ? 1 : 0)) continue;
    float vx, vy, ox, oy;
    if (f == 0) vel_cell(vs, ci, cj, vx, vy);
    else if (f == 1) vel_uface(vs, ci, cj, vx, vy);
    else vel_vface(vs, ci, cj, vx, vy);
    const float hx = vs.bounded(hd * vx), hy = vs.bounded(hd * vy);
    trace_from(vs, (float)ci + (f == 1 ? 0.f : 0.5f), (float)cj + (f == 2 ? 0.f : 0.5f), hx, hy, dt, ox, oy);
    if (f == 0) {
      const int r = (b + H) * RW + a + H;
      sTh[r] = sample(Tf, ox, oy, 0.5f, 0.5f);
      sYh[r] = sample4(Yf, ox, oy);
    } else if (f == 1) {
      sUh[(b + H) * UW + a + H] = sample(vs.u, ox, oy, 0.f, 0.5f);
    } else {
      sVh[(b + H) * VW + a + H] = sample(vs.v, ox, oy, 0.5f, 0.f);
    }
  }
  __syncthreads();

  // the lookups' region is the widest one: with h < H no correction of the tile's own sites reads beyond h cells
  const ThLookup Th{sTh, rx0, ry0, RW, RH, &S, &Tf};
  const YhLookup Yh{sYh, rx0, ry0, RW, RH, &S, &Yf};
  const UhLookup Uh{sUh, rx0, ry0, UW, UH, UW, &S, &vs};
  const VhLookup Vh{sVh, rx0, ry0, VW, VH, VW, &S, &vs};
  if (own) {
    // ---- scalCorrect (advect.wgsl:78-103)
    const float sO2 = S.P.sO2;
    const int k = j * pc + i;
    float tx, ty;
    const int bi = floor_frac(cbx - 0.5f, tx), bj = floor_frac(cby - 0.5f, ty);
    float A, C, D, E;
    corners(Th, bi, bj, A, C, D, E);
    const float Tc = th + 0.5f * (__ldg(S.T + k) - mixf(mixf(A, C, tx), mixf(D, E, tx), ty));
    const float4 y0v = __ldg(S.Y + k);
    float4 A4, C4, D4, E4;
    corners(Yh, bi, bj, A4, C4, D4, E4);
    const float4 sb = mix4(mix4(A4, C4, tx), mix4(D4, E4, tx), ty);
    const float4 Yc = make_float4(yh.x + 0.5f * (y0v.x - sb.x), yh.y + 0.5f * (y0v.y - sb.y),
                                  yh.z + 0.5f * (y0v.z - sb.z), yh.w + 0.5f * (y0v.w - sb.w));
    const bool inT = Tc >= tlo && Tc <= thi;
    const bool inY = Yc.x >= ylo.x && Yc.y >= ylo.y && Yc.z >= ylo.z && Yc.w >= ylo.w &&
                     Yc.x <= yhi.x && Yc.y <= yhi.y && Yc.z <= yhi.z && Yc.w <= yhi.w;
    const float mixC = fminf(Yc.x, Yc.y / sO2);
    const float mixL = fminf(yh.x, yh.y / sO2);
    if (inT && inY && mixC <= mixL + 1e-5f) { S.T2[k] = Tc; S.Y2[k] = Yc; }
    else { S.T2[k] = th; S.Y2[k] = yh; }
    // ---- velCorrect (advect.wgsl:52-65)
    S.U2[j * pu + i] = clampf(uh + 0.5f * (__ldg(S.U + j * pu + i) - sample(Uh, ubx, uby, 0.f, 0.5f)), ulo, uhi);
    S.V2[k] = clampf(vh + 0.5f * (__ldg(S.V + k) - sample(Vh, vbx, vby, 0.5f, 0.f)), vlo, vhi);
  }
  if (!last) return;
  // ---- the domain's last faces, x = nx and y = ny. They may travel farther than the tile's own sites, whose
  // reach alone set the staged width, so their lookups' region is the staged one: values beyond it are
  // recomputed. (Their reach traced before the barrier instead: +0.8 us per step at 32x48, +1 at 160x224.)
  const int hs = s_h;
  if (x0 + TX >= nx && threadIdx.x < TY && y0 + (int)threadIdx.x < ny) {
    const int fj = y0 + threadIdx.x, k = fj * pu + nx;
    const float gx = (float)nx, gy = (float)fj + 0.5f;
    float ox, oy, lo, hi; vs.trace(gx, gy, dt, ox, oy);
    const float h1 = sample_range(vs.u, ox, oy, 0.f, 0.5f, lo, hi);
    vs.trace(gx, gy, -dt, ox, oy);
    const UhLookup Ul{sUh + (H - hs) * (UW + 1), x0 - hs, y0 - hs, TX + 2 * hs + 1, TY + 2 * hs, UW, &S, &vs};
    S.U2[k] = clampf(h1 + 0.5f * (__ldg(S.U + k) - sample(Ul, ox, oy, 0.f, 0.5f)), lo, hi);
  }
  if (y0 + TY >= ny && threadIdx.x >= NT - TX && x0 + li < nx) {
    const int k = ny * pc + i;
    const float gx = (float)i + 0.5f, gy = (float)ny;
    float ox, oy, lo, hi; vs.trace(gx, gy, dt, ox, oy);
    const float h1 = sample_range(vs.v, ox, oy, 0.5f, 0.f, lo, hi);
    vs.trace(gx, gy, -dt, ox, oy);
    const VhLookup Vl{sVh + (H - hs) * (VW + 1), x0 - hs, y0 - hs, TX + 2 * hs, TY + 2 * hs + 1, VW, &S, &vs};
    S.V2[k] = clampf(h1 + 0.5f * (__ldg(S.V + k) - sample(Vl, ox, oy, 0.5f, 0.f)), lo, hi);
  }
}

void launch_advect(const SceneDesc* scenes, const Work* work, int ntiles, int shape, cudaStream_t st) {
  if (ntiles <= 0) return;
  static_assert(TILE_TX[0] == ADV_TX && TILE_TY[0] == ADV_TY, "shape 0 is the default tile");
  if (shape == 1) k_advect<TILE_TX[1], TILE_TY[1], ADV_H><<<ntiles, TILE_TX[1] * TILE_TY[1], 0, st>>>(scenes, work);
  else if (shape == 2) k_advect<TILE_TX[2], TILE_TY[2], ADV_H><<<ntiles, TILE_TX[2] * TILE_TY[2], 0, st>>>(scenes, work);
  else k_advect<ADV_TX, ADV_TY, ADV_H><<<ntiles, ADV_TX * ADV_TY, 0, st>>>(scenes, work);
}

}  // namespace cfg
