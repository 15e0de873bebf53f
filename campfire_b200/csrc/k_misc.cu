// Projection (pressure.wgsl:159-180), the CFL step update, geometry
// rasterisation (geometry.wgsl), radiation to wood faces (radiation.wgsl) and
// the FP64 budget sums.
#include "gas_dev.cuh"
#include "kernels.h"
#include "reduce.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace cfg {

// u -= dt (1/rho_f) grad p; ghost -p at the open sides/top, closed faces 0.
// FP64: the FP64 pressure of the defect-correction loop, rounded once to f32.
// CFL step for the next step: dt = min(dt_cap, cfl*dx/max|u|) and the diffusion
// sub-step count of js/fluid.js:190-198 for that dt (one thread, after max|u| is complete)
// advance_clock: the step's own dt (P.dt, before it is replaced) is added to the scene's clock
__device__ __forceinline__ void cfl_next_dt(SceneDesc& S, double h, double alpha, bool advance_clock) {
  if (advance_clock) S.solve->time += (double)S.P.dt;
  const float m = __uint_as_float(S.solve->maxu);
  const float cand = m > 0.f ? S.cfl * S.P.dx / m : S.dt_cap;
  const float dt = fminf(S.dt_cap, cand);
  S.P.dt = dt;
  int n = (int)ceil((double)dt / (h * h / (4.5 * alpha)));
  n = min(5, n % 2 ? n : n + 1);
  S.diff_sub = n;
  S.diff_dt = (float)((double)dt / n);
  S.solve->maxu = 0u;
}

// post (the step's tail folded into the projection): bit 0 swaps every scene's coarsest
// inverse halves (after the factorisation's branch has joined), bit 1 sets each CFL scene's
// next dt in the scene's last CTA (arrival on the scene's counter after its max|u|).
// Bound by latency: one cell per thread, and a chain of L2 loads and quotients. What the cell's two
// faces need is requested together whatever the faces' open fractions (before, the V face waited
// for the U face, and each for its open fraction), and the quotients by rhoAmb Tamb and dx come
// from reciprocals formed once per CTA: a step of 224x320 86.7 -> 85.9 us, of 256x384 268.1 -> 266.4, of the
// 64-scene batch 3784 -> 3762.
template <bool FP64>
__global__ void __launch_bounds__(256) k_project(SceneDesc* __restrict__ scenes, const Work* __restrict__ work, int nscenes,
                                                 int post, const double* dxd, const double* alpha, float* dtv) {
  __shared__ float redm[32];
  __shared__ int s_last;
  const Work w = work[blockIdx.x];
  if ((post & 1) && blockIdx.x == 0)
    for (int s = threadIdx.x; s < nscenes; s += blockDim.x) {
      const SceneDesc& Q = scenes[s];
      if (!Q.enabled) continue;
      SolveState* ss = Q.solve;
      ss->cinv_cur ^= 1;
      ss->direct_ok = ss->direct_ok_next;
      ss->direct_ok_next = 0;
    }
  SceneDesc& S = scenes[w.scene];
  if (!S.enabled) return;
  const cfg_params& P = S.P;
  const int nx = S.nx, ny = S.ny, pc = S.pc, pu = S.pu;
  const LevelDesc L0 = S.lev[0];
  const float* p = L0.p;
  const double* p64 = S.p64;
  const float dt = P.dt, dx = P.dx, rT = P.rhoAmb * P.Tamb;
  const int i = w.tx * PR_TX + (threadIdx.x % PR_TX), j = w.ty * PR_TY + (threadIdx.x / PR_TX);
  // the west U face and the south V face of the cell
  using real = typename std::conditional<FP64, double, float>::type;
  __shared__ real s_r[2];
  const bool in = i < nx && j < ny;
  float* const U = S.U;
  float* const V = S.V;
  float fu = 0.f, fv = 0.f, u0 = 0.f, v0 = 0.f, T0 = 0.f, Tw = 0.f, Ts = 0.f;
  real p0 = 0, pw = 0, ps = 0;
  if (in) {
    const int iw = max(i - 1, 0), js = max(j - 1, 0);
    auto at = [&](int a, int b) -> real { if constexpr (FP64) return p64[b * nx + a]; else return p[b * L0.pc + a]; };
    fu = __ldg(S.fx + j * pu + i); fv = __ldg(S.fy + j * pc + i);
    u0 = U[j * pu + i]; v0 = V[j * pc + i];
    T0 = __ldg(S.T + j * pc + i); Tw = __ldg(S.T + j * pc + iw); Ts = __ldg(S.T + js * pc + i);
    p0 = at(i, j); pw = at(iw, j); ps = at(i, js);
  }
  if (threadIdx.x == 0) { s_r[0] = (real)1 / (real)rT; s_r[1] = (real)1 / (real)dx; }
  __syncthreads();
  const real rr = s_r[0], rx = s_r[1];
  // face velocity from its own, the mean temperature, and the pressures behind and ahead
  auto face = [&](float f, float w, float Ta, float Tb, real pa, real pb) {
    if (!(f > 0.f)) return 0.f;
    if constexpr (FP64) {
      const double Tf = 0.5 * ((double)Ta + (double)Tb);
      const double x = (double)dt * ddiv_by_rcp(Tf, (double)rT, rr) * (pb - pa);
      return (float)((double)w - (fabs(x) < 1e290 ? ddiv_by_rcp(x, (double)dx, rx) : x / (double)dx));
    } else {
      const float Tf = 0.5f * (Ta + Tb);
      const float x = dt * div_by_rcp(Tf, rT, rr) * (pb - pa), a = fabsf(x);
      return w - (a > 1e-30f && a < 1e30f ? div_by_rcp(x, dx, rx) : x / dx);
    }
  };
  auto pf = [&](int a, int b) { return p[b * L0.pc + a]; };
  auto pd = [&](int a, int b) { return p64[b * nx + a]; };
  auto Tat = [&](int a, int b) { return __ldg(S.T + b * pc + a); };
  float m = 0.f;
  auto uface = [&](int a, int b) {
    const int k = b * pu + a;
    float u;
    if (__ldg(S.fx + k) > 0.f) {
      if (FP64) {
        const double Tf = 0.5 * ((double)Tat(min(max(a - 1, 0), nx - 1), b) + (double)Tat(min(a, nx - 1), b));
        const double pl = a > 0 ? pd(a - 1, b) : -pd(0, b);
        const double pr = a < nx ? pd(min(a, nx - 1), b) : -pd(nx - 1, b);
        u = (float)((double)S.U[k] - (double)dt * (Tf / (double)rT) * (pr - pl) / (double)dx);
      } else {
        const float Tf = 0.5f * (Tat(min(max(a - 1, 0), nx - 1), b) + Tat(min(a, nx - 1), b));
        const float pl = a > 0 ? pf(max(a - 1, 0), b) : -pf(0, b);
        const float pr = a < nx ? pf(min(a, nx - 1), b) : -pf(nx - 1, b);
        u = S.U[k] - dt * (Tf / rT) * (pr - pl) / dx;
      }
    } else u = 0.f;
    S.U[k] = u;
    m = fmaxf(m, fabsf(u));
  };
  auto vface = [&](int a, int b) {
    const int k = b * pc + a;
    float v;
    if (b > 0 && __ldg(S.fy + k) > 0.f) {
      if (FP64) {
        const double Tf = 0.5 * ((double)Tat(a, b - 1) + (double)Tat(a, min(b, ny - 1)));
        const double pb = pd(a, b - 1);
        const double pt = b < ny ? pd(a, min(b, ny - 1)) : -pd(a, ny - 1);
        v = (float)((double)S.V[k] - (double)dt * (Tf / (double)rT) * (pt - pb) / (double)dx);
      } else {
        const float Tf = 0.5f * (Tat(a, b - 1) + Tat(a, min(b, ny - 1)));
        const float pb = pf(a, b - 1);
        const float pt = b < ny ? pf(a, min(b, ny - 1)) : -pf(a, ny - 1);
        v = S.V[k] - dt * (Tf / rT) * (pt - pb) / dx;
      }
    } else v = 0.f;
    S.V[k] = v;
    m = fmaxf(m, fabsf(v));
  };
  if (in) {
    const float u = face(fu, u0, Tw, T0, i > 0 ? pw : -p0, p0), v = j > 0 ? face(fv, v0, Ts, T0, ps, p0) : 0.f;
    U[j * pu + i] = u;
    V[j * pc + i] = v;
    m = fmaxf(fmaxf(m, fabsf(u)), fabsf(v));
    // the domain's east and north faces
    if (i == nx - 1) uface(nx, j);
    if (j == ny - 1) vface(i, ny);
  }
  const float bm = block_max(m, redm);
  if (threadIdx.x == 0 && S.cfl > 0.f) atomicMax(&S.solve->maxu, __float_as_uint(bm));
  if (!(post & 2) || !(S.cfl > 0.f)) return;
  // every CTA of the scene has read P.dt and added its max|u| before it arrives
  if (threadIdx.x == 0) s_last = arrive_acq_rel(&S.solve->counter) == (unsigned)S.nt_mg0 - 1u;
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    S.solve->counter = 0u;
    cfl_next_dt(S, dxd[w.scene], alpha[w.scene], true);
    if (dtv) {   // pinned host memory: visible to the host once the step's event has passed
      dtv[w.scene] = S.P.dt;
      __threadfence_system();
    }
  }
}

// the CFL update on its own (one thread per scene)
__global__ void k_cfl_update(SceneDesc* scenes, int nscenes, const double* dxd, const double* alpha) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nscenes) return;
  SceneDesc& S = scenes[s];
  if (!S.enabled || !(S.cfl > 0.f)) return;
  cfl_next_dt(S, dxd[s], alpha[s], false);
}

// geometry.wgsl:121-153: per cell the nearest piece (sdf, piece*4+face) and the
// band weight; per face the open fraction. Tiles cover (nx+1) x (ny+1) sites.
// Each tile first keeps the pieces that can be the nearest of any of its sites, in order (a
// piece farther from the tile's centre than another by more than the tile's diameter cannot),
// and each piece's rotation is evaluated once per tile instead of at every site: bound by the
// sites' arithmetic, 3 sites x the pieces that are left. 22.1 -> 8.4 us
// at 224x320 with 16 pieces, 82 -> 10.4 us at 352x512 with 40.
namespace {
// common.wgsl:47-62, the signed distance to a rotated square (negative inside) and its nearest face
// (0: +x, 1: +y, 2: -x, 3: -y), with the rotation's cosine and sine at hand
struct RotPiece { float x, y, half, c, s; int n; };
__device__ __forceinline__ float sd_rot(float px, float py, const RotPiece& q, float& lx, float& ly) {
  const float dxp = px - q.x, dyp = py - q.y;
  lx = q.c * dxp + q.s * dyp; ly = -q.s * dxp + q.c * dyp;
  const float qx = fabsf(lx) - q.half, qy = fabsf(ly) - q.half;
  const float mx = fmaxf(qx, 0.f), my = fmaxf(qy, 0.f);
  return sqrtf(mx * mx + my * my) + fminf(fmaxf(qx, qy), 0.f);
}
}  // namespace
__global__ void __launch_bounds__(256) k_geometry(const SceneDesc* __restrict__ scenes, const Work* __restrict__ work) {
  __shared__ RotPiece sp[MAX_PIECES];
  __shared__ int s_np;
  const Work w = work[blockIdx.x];
  const SceneDesc& S = scenes[w.scene];
  if (!S.enabled) return;
  const cfg_params& P = S.P;
  const int np = min(max(P.nPieces, 0), MAX_PIECES);
  const float dx = P.dx;
  if (threadIdx.x < 32) {
    // lower and upper bounds of each piece's distance over the tile (radius r about its
    // centre, half a cell more than its sites reach): a square of half side h lies between the
    // discs of radius h and 1.5 h; 1e-4 of the lengths covers the rounding of both evaluations
    const float cx = ((float)(w.tx * GEO_TX) + 0.5f * GEO_TX) * dx, cy = ((float)(w.ty * GEO_TY) + 0.5f * GEO_TY) * dx;
    const float r = 0.5f * sqrtf((float)((GEO_TX + 2) * (GEO_TX + 2) + (GEO_TY + 2) * (GEO_TY + 2))) * dx;
    const Piece* pcs = reinterpret_cast<const Piece*>(S.pieces);
    RotPiece q[2];
    bool on[2];
    float lo[2], up = 3e38f;
    #pragma unroll
    for (int k = 0; k < 2; k++) {
      const int n = threadIdx.x + 32 * k;
      on[k] = n < np && !(pcs[n].alive <= 0.f);
      if (!on[k]) continue;
      const Piece& pc = pcs[n];
      q[k] = RotPiece{pc.pos[0], pc.pos[1], pc.half, cosf(pc.angle), sinf(pc.angle), n};
      const float ex = cx - q[k].x, ey = cy - q[k].y, d = sqrtf(ex * ex + ey * ey), h = fabsf(q[k].half);
      const float eps = 1e-4f * (d + r + h);
      lo[k] = d - r - 1.5f * h - eps;
      up = fminf(up, d + r + (q[k].half < 0.f ? 3.f * h : -h) + eps);
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) up = fminf(up, __shfl_xor_sync(0xffffffffu, up, o));
    int cnt = 0;
    #pragma unroll
    for (int k = 0; k < 2; k++) {
      const bool keep = on[k] && !(lo[k] > up);
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) sp[cnt + __popc(m & ((1u << threadIdx.x) - 1u))] = q[k];
      cnt += __popc(m);
    }
    if (threadIdx.x == 0) s_np = cnt;
  }
  __syncthreads();
  const int nk = s_np;
  const int nx = S.nx, ny = S.ny;
  const int i = w.tx * GEO_TX + (threadIdx.x % GEO_TX), j = w.ty * GEO_TY + (threadIdx.x / GEO_TX);
  auto nearest = [&](float px, float py) {
    float best = 1e9f;
    for (int n = 0; n < nk; n++) {
      float lx, ly;
      const float d = sd_rot(px, py, sp[n], lx, ly);
      if (d < best) best = d;
    }
    return best;
  };
  if (i < nx && j < ny) {
    const float px = ((float)i + 0.5f) * dx, py = ((float)j + 0.5f) * dx;
    float best = 1e9f;
    uint32_t bid = SOLID_NONE;
    for (int n = 0; n < nk; n++) {
      float lx, ly;
      const float d = sd_rot(px, py, sp[n], lx, ly);
      if (d < best) {
        best = d;
        const uint32_t face = fabsf(lx) > fabsf(ly) ? (lx > 0.f ? 0u : 2u) : (ly > 0.f ? 1u : 3u);
        bid = (uint32_t)sp[n].n * 4u + face;
      }
    }
    S.cellG[j * S.pc + i] = make_float2(best, __uint_as_float(bid));
    if (bid != SOLID_NONE && best >= 0.f && best < 2.f * dx) {
      const float wgt = fmaxf(0.f, 1.f - fabsf(best - dx) / dx) / dx;
      atomicAdd(S.faceW + bid, wgsl_i32_round(wgt * dx * dx * 1.0e8f));
    }
  }
  if (i <= nx && j < ny) {
    const float d = nearest((float)i * dx, ((float)j + 0.5f) * dx);
    S.fx[j * S.pu + i] = clampf(0.5f + d / dx, 0.f, 1.f);
  }
  if (i < nx && j <= ny) {
    const float d = nearest(((float)i + 0.5f) * dx, (float)j * dx);
    S.fy[j * S.pc + i] = j == 0 ? 0.f : clampf(0.5f + d / dx, 0.f, 1.f);
  }
}

// ---------------------------------------------------------------- radiation.wgsl
namespace {
__device__ __forceinline__ float planck580(float t) {   // :28-33
  const float l = 580e-9f;
  const float x = 1.438777e-2f / (l * t);
  if (x > 80.f) return 0.f;
  return 1.191042e-16f / (l * l * l * l * l) / (expf(x) - 1.f) * 1e-9f;
}
// :36-51 ray vs rotated box: t_enter (or < 0) and the face hit; c, s: the piece's rotation
__device__ __forceinline__ void hitBox(float ox, float oy, float dxr, float dyr, const Piece& pc, float c, float s,
                                       float& tn_out, float& face) {
  const float qx = ox - pc.pos[0], qy = oy - pc.pos[1];
  const float lox = c * qx + s * qy, loy = -s * qx + c * qy;
  const float ldx = c * dxr + s * dyr, ldy = -s * dxr + c * dyr;
  const float h = pc.half;
  const float invx = 1.f / (fabsf(ldx) < 1e-9f ? 1e-9f : ldx);
  const float invy = 1.f / (fabsf(ldy) < 1e-9f ? 1e-9f : ldy);
  const float t1x = (-h - lox) * invx, t1y = (-h - loy) * invy;
  const float t2x = (h - lox) * invx, t2y = (h - loy) * invy;
  const float tminx = fminf(t1x, t2x), tminy = fminf(t1y, t2y);
  const float tmaxx = fmaxf(t1x, t2x), tmaxy = fmaxf(t1y, t2y);
  const float tn = fmaxf(tminx, tminy), tf = fminf(tmaxx, tmaxy);
  if (tf < 0.f || tn > tf || tn < 1e-5f) { tn_out = -1.f; face = 0.f; return; }
  if (tminx > tminy) face = ldx < 0.f ? 0.f : 2.f; else face = ldy < 0.f ? 1.f : 3.f;
  tn_out = tn;
}
__device__ __forceinline__ float fractf(float x) { return x - floorf(x); }
}  // namespace

// gasAt (:53-62) of every cell: emission towards a ray and its visible share. A ray samples
// the cell under each of its points, so the pair is a function of the cell alone; evaluated
// once per cell (20 B read, 8 B written) it leaves each of the 1-3 million ray samples one 8-byte
// gather. The pair goes to the scene's spare species array Yw.
__global__ void __launch_bounds__(256) k_emission(const SceneDesc* __restrict__ scenes, int scene) {
  const SceneDesc& S = scenes[scene];
  const cfg_params& P = S.P;
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (i >= S.nx || j >= S.ny) return;
  const int k = j * S.pc + i;
  const float T4a = powf(P.Tamb, 4.f);
  const float Tg = __ldg(S.T + k); const float4 Yg = __ldg(S.Y + k);
  const float fv = rhoOf(P, Tg) * Yg.w / P.sootDensity;
  const float kap = P.kappaSootC * fv * Tg + P.kappaGas * Yg.z;
  const float T2v = Tg * Tg;
  reinterpret_cast<float2*>(S.Yw)[k] =
      make_float2(kap * P.sigma * (T2v * T2v - T4a) / 3.14159265f, 6.3f * fv / 580e-9f * planck580(Tg));
}

// :64-158 a cluster of CTAs per wood face or floor probe, RAD_RT rays at a time each (1024 rays are the
// most; up to RAD_CL CTAs share them). The rays of a CTA go through the same phases
// together, once for the way from their origin and once after the floor's bounce: (1) the first
// piece hit, G lanes per ray sharing the pieces; (2) the samples along the rays, RAD_CH per ray at
// a time, by all warps but the last, which at the same time (3) adds the chunk before to its rays'
// sums in the order of the reference's loop. The first CTA adds the rays' shares in the
// reference's tree. Bound by instruction issue and by the spread of the rays' lengths over the
// SMs: one thread per ray marching its samples alone was two warps per SM in a serial chain of
// 200-600 samples, one CTA of 1024 threads per target left the longest targets' SMs last.
// With 64 rays and 16 pieces: 453 -> 29 us at 224x320 (35 with a CTA per target); 40 pieces at
// 352x512: 721 -> 50 us (55); k_emission's 7 us included.
namespace {
constexpr int RAD_CH = 64, RAD_THREADS = 256, RAD_CL = 8;
constexpr int RAD_ROW = RAD_CH + 1;   // terms of a ray in shared memory: odd, so that a warp of rays reads 32 banks
struct Ray { float ox, oy, dx, dy, tOut, tFloor, rns, hitT; int ns, next; };   // next: 0 done, 1 bounces
}
template <int RAD_RT>
__global__ void __launch_bounds__(RAD_THREADS) k_radiation(const SceneDesc* __restrict__ scenes, int scene, int NRAY) {
  __shared__ __align__(16) float2 terms[2 * RAD_RT * RAD_ROW];
  __shared__ Piece sp[MAX_PIECES];
  __shared__ float sc[MAX_PIECES], ss[MAX_PIECES];
  __shared__ float sq[1024], sv[1024];
  __shared__ Ray ray[RAD_RT];
  __shared__ int s_max;
  const SceneDesc& S = scenes[scene];
  const cfg_params& P = S.P;
  const int np = min(max(P.nPieces, 0), MAX_PIECES);
  for (int e = threadIdx.x; e < np * PIECE_FLOATS; e += blockDim.x)
    reinterpret_cast<float*>(sp)[e] = S.pieces[e];
  __syncthreads();
  if ((int)threadIdx.x < np) { sc[threadIdx.x] = cosf(sp[threadIdx.x].angle); ss[threadIdx.x] = sinf(sp[threadIdx.x].angle); }
  __syncthreads();
  const float PI = 3.14159265f;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int ncta = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const uint32_t tgt = blockIdx.x / ncta;
  const uint32_t nFaces = (uint32_t)np * 4u;
  const int nx = S.nx, ny = S.ny, pcw = S.pc;
  const float dx = P.dx, rdx = __frcp_rn(dx);
  const float2* E = reinterpret_cast<const float2*>(S.Yw);
  const bool face = tgt < nFaces;
  const bool valid = face ? sp[tgt / 4u].alive > 0.f : tgt - nFaces < (uint32_t)N_FLOOR;
  if (!valid) return;   // the same in every thread of the cluster: nothing of this target is written
  cl.sync();            // every CTA runs: the first one's shared memory may be written
  const int RT = min(NRAY, RAD_RT);
  const int G = min(RAD_THREADS / RT, 32);   // lanes per ray in phase 1 (both powers of two)
  const int tid = threadIdx.x, sum0 = RAD_THREADS - 32;   // the last warp adds
  for (int r0 = rank * RT; r0 < NRAY; r0 += ncta * RT) {
    float J = 0.f, Jv = 0.f, Twall = P.Tamb, cosn = 0.f;   // of ray r0 + tid - sum0 in the adding threads
    const int mine = tid - sum0;
    if (mine >= 0 && mine < RT) {
      const uint32_t li = (uint32_t)(r0 + mine);
      float nrx = 0.f, nry = 1.f;
      Ray q;
      if (face) {
        const Piece& pc = sp[tgt / 4u];
        const uint32_t f = tgt % 4u;
        const float c = sc[tgt / 4u], s = ss[tgt / 4u];
        float lnx = 1.f, lny = 0.f;
        if (f == 1u) { lnx = 0.f; lny = 1.f; } else if (f == 2u) { lnx = -1.f; lny = 0.f; } else if (f == 3u) { lnx = 0.f; lny = -1.f; }
        nrx = c * lnx - s * lny; nry = s * lnx + c * lny;
        const float tx = -nry, ty = nrx;
        const float u = (fractf((float)li * 0.618034f + (float)P.frame * 0.1234f) - 0.5f) * 1.6f * pc.half;
        const float hh = pc.half + 1e-4f;
        q.ox = pc.pos[0] + nrx * hh + tx * u; q.oy = pc.pos[1] + nry * hh + ty * u;
      } else {
        q.ox = ((float)(tgt - nFaces) + 0.5f) / (float)N_FLOOR * (float)P.nx * dx; q.oy = 1e-4f;
      }
      const float jit = fractf((float)P.frame * 0.7548777f + (float)tgt * 0.5698403f);
      const float a = (((float)li + jit) / (float)NRAY - 0.5f) * PI;
      cosn = cosf(a);
      const float base = atan2f(nry, nrx);
      q.dx = cosf(base + a); q.dy = sinf(base + a);
      q.next = 1;
      ray[mine] = q;
    }
    for (int leg = 0; leg < 2; leg++) {
      if (tid == 0) s_max = 0;
      __syncthreads();
      // ---- (1) the leg's end: first piece in the reference's order (the nearest, the lower index
      // among equals), floor, domain
      if (tid < RT * G) {
        const int r = tid / G, g = tid & (G - 1);
        const float ox = ray[r].ox, oy = ray[r].oy, ddx = ray[r].dx, ddy = ray[r].dy;
        const bool live = ray[r].next != 0;
        float tHit = 1e9f, hitT = 0.f;
        int hitN = MAX_PIECES;
        if (live)
          for (int n = g; n < np; n += G) {
            const Piece& pc = sp[n];
            if (pc.alive <= 0.f) continue;
            float hx, hy; hitBox(ox, oy, ddx, ddy, pc, sc[n], ss[n], hx, hy);
            if (hx > 0.f && hx < tHit) { tHit = hx; hitT = pc.Ts[(uint32_t)hy]; hitN = n; }
          }
        // whole warps are here (RT G is a multiple of 32 for every power of two of rays): the full mask brings
        // the lanes together again that left the loop over the pieces at different turns
        for (int o = G / 2; o > 0; o >>= 1) {
          const float t2 = __shfl_xor_sync(0xffffffffu, tHit, o), T2 = __shfl_xor_sync(0xffffffffu, hitT, o);
          const int n2 = __shfl_xor_sync(0xffffffffu, hitN, o);
          if (t2 < tHit || (t2 == tHit && n2 < hitN)) { tHit = t2; hitT = T2; hitN = n2; }
        }
        if (g == 0) {
          int ns = 0, next = 0;
          float tOut = 0.f, tFloor = 1e9f, wallT = P.Tamb;
          if (live) {
            if (ddy < -1e-6f) tFloor = -oy / ddy;
            const float tEnd = fminf(tHit, tFloor);
            const float W = (float)P.nx * dx, H = (float)P.ny * dx;
            float tx = 1e9f, ty = 1e9f;
            if (ddx > 1e-6f) tx = (W - ox) / ddx; else if (ddx < -1e-6f) tx = -ox / ddx;
            if (ddy > 1e-6f) ty = (H - oy) / ddy;
            tOut = fminf(fminf(tx, ty), tEnd);
            ns = max(wgsl_i32(ceilf(tOut / dx)), 0);
            if (tHit < tFloor && tHit < 1e8f) wallT = hitT;
            else if (tFloor < 1e8f && tFloor <= tHit && leg == 0) next = 1;
          }
          Ray& q = ray[r];
          // a ray that ended on the first leg keeps its wall temperature
          q.tOut = tOut; q.tFloor = tFloor; q.rns = __frcp_rn((float)ns); q.ns = ns;
          if (live) { q.hitT = wallT; q.next = next; }
          atomicMax(&s_max, ns);
        }
      }
      __syncthreads();
      // ---- (2) and (3): chunk k is evaluated while chunk k - 1 is added
      const int chunks = s_max / RAD_CH + (s_max % RAD_CH != 0);
      for (int k = 0; k <= chunks; k++) {
        if (tid < sum0) {
          if (k < chunks) {
            float2* buf = terms + (size_t)(k & 1) * RAD_RT * RAD_ROW;
            for (int e = tid; e < RT * RAD_CH; e += sum0) {
              const int r = e / RAD_CH, m = k * RAD_CH + e % RAD_CH;
              const Ray& q = ray[r];
              if (m >= q.ns) continue;
              const float fns = (float)q.ns;
              // quotients by the sample count and the cell size by their reciprocals: the IEEE ones
              const float t = div_by_rcp(((float)m + 0.5f) * q.tOut, fns, q.rns);
              const float px = q.ox + q.dx * t, py = q.oy + q.dy * t;
              const int gi = wgsl_i32(div_by_rcp(px, dx, rdx)), gj = wgsl_i32(div_by_rcp(py, dx, rdx));
              float2 g = make_float2(0.f, 0.f);
              if (!(gi < 0 || gj < 0 || gi >= nx || gj >= ny)) g = E[gj * pcw + gi];
              // emission fades to nothing in clear air: its quotients stay exact
              buf[r * RAD_ROW + e % RAD_CH] = make_float2(div_tiny(g.x * q.tOut, fns, q.rns), div_tiny(g.y * q.tOut, fns, q.rns));
            }
          }
        } else if (k > 0 && mine < RT) {
          const float2* row = terms + (size_t)((k - 1) & 1) * RAD_RT * RAD_ROW + mine * RAD_ROW;
          const int cnt = min(ray[mine].ns - (k - 1) * RAD_CH, RAD_CH);
          #pragma unroll 8
          for (int m = 0; m < cnt; m++) { const float2 g = row[m]; J += g.x; Jv += g.y; }
        }
        __syncthreads();
      }
      if (mine >= 0 && mine < RT) {
        Ray& q = ray[mine];
        if (q.next) {   // off the floor
          q.ox = q.ox + q.dx * q.tFloor; q.oy = q.oy + q.dy * q.tFloor + 1e-5f;
          q.dy = -q.dy;
        }
      }
      __syncthreads();
    }
    if (mine >= 0 && mine < RT) {
      Twall = ray[mine].hitT;
      const float wgt = PI / (float)NRAY * cosn;
      const float T2v = Twall * Twall;
      cl.map_shared_rank(sq, 0)[r0 + mine] = wgt * (0.5f * P.sigma * T2v * T2v + 2.f * J);
      cl.map_shared_rank(sv, 0)[r0 + mine] = wgt * (2.f * Jv);
    }
  }
  cl.sync();
  if (rank != 0) return;
  const int li = tid;
  for (int s = NRAY / 2; s > 0; s >>= 1) {
    for (int k = li; k < s; k += RAD_THREADS) { sq[k] += sq[k + s]; sv[k] += sv[k + s]; }
    __syncthreads();
  }
  if (li == 0) {
    const float4 old = S.rad[tgt];
    const float al = old.x <= 0.f ? 1.f : 0.35f;
    S.rad[tgt] = make_float4(mixf(old.x, sq[0], al), mixf(old.y, sv[0], al), 0.f, 0.f);
  }
}

// FP64 budgets over gas cells of one scene: seven sums and the largest temperature (as k_residual_norms:
// partials per CTA, added by the last one). The call, result on the host: 366 -> 33 us at 512x768.
__global__ void __launch_bounds__(256) k_budgets(const SceneDesc* __restrict__ scenes, int scene, double* out) {
  __shared__ double sh[7 * 257];
  __shared__ float redm[32];
  const SceneDesc& S = scenes[scene];
  const cfg_params& P = S.P;
  const double cellA = (double)P.dx * (double)P.dx;
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  float tmax = 0.f;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < S.nx * S.ny; e += gridDim.x * blockDim.x) {
    const int i = e % S.nx, j = e / S.nx, k = j * S.pc + i;
    const float2 g = S.cellG[k];
    if (g.x < 0.f && __float_as_uint(g.y) != SOLID_NONE) continue;
    const double t = (double)S.T[k];
    const double rho = (double)P.rhoAmb * (double)P.Tamb / t;
    const float4 y = S.Y[k];
    v[0] += rho * cellA; v[1] += rho * (double)P.cp * t * cellA;
    v[2] += rho * (double)y.x * cellA; v[3] += rho * (double)y.y * cellA;
    v[4] += rho * (double)y.z * cellA; v[5] += rho * (double)y.w * cellA;
    v[6] += (double)S.SQ[k].y * cellA;
    tmax = fmaxf(tmax, S.T[k]);
  }
  const float bm = block_max(tmax, redm);
  // the CTA's maximum past every CTA's seven sums, published by the same arrival
  if (threadIdx.x == 0) S.part[7 * gridDim.x + blockIdx.x] = (double)bm;
  block_sum_t<7>(v, sh);
  if (!scene_reduce_n<7>(S, blockIdx.x, gridDim.x, v, sh)) return;
  float tm = 0.f;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) tm = fmaxf(tm, (float)__ldcg(S.part + 7 * gridDim.x + k));
  tm = block_max(tm, redm);
  if (threadIdx.x == 0) {
    #pragma unroll
    for (int q = 0; q < 7; q++) out[q] = v[q];
    out[7] = (double)tm;
  }
}

// ------------------------------------------------------------------ host blocks by value, readback
// A scene's parameter block (writeParams, js/fluid.js:180-199) and its pieces (uploadPieces,
// js/fluid.js:201-204) arrive as kernel parameters: one launch each instead of copy-engine
// transfers beside the compute stream, and the host's copy is free again once the launch returns.
// k_write_params leaves out word `skip` and words [s0, s1) (the step-owned dt and diffusion
// sub-steps of a CFL scene; -1: none).
__global__ void k_write_params(uint32_t* __restrict__ dst, const ParamWords b, int skip, int s0, int s1) {
  for (int k = threadIdx.x; k < PARAM_WORDS; k += blockDim.x)
    if (k != skip && (k < s0 || k >= s1)) dst[k] = b.w[k];
}
__global__ void k_write_pieces(float* __restrict__ dst, const PieceFloats b) {
  for (int k = threadIdx.x; k < MAX_PIECES * PIECE_FLOATS; k += blockDim.x) dst[k] = b.f[k];
}
// The readback (js/fluid.js:315-342): nwords words from src into pinned host memory mapped into the
// device's address space, then the first nzero of them (the accumulators) cleared on the device;
// each thread clears only words it has read. The host reads the slot after the event that follows.
__global__ void k_readback(uint32_t* __restrict__ src, uint32_t* __restrict__ host, int nwords, int nzero) {
  for (int k = threadIdx.x; k < nwords; k += blockDim.x) {
    host[k] = src[k];
    if (k < nzero) src[k] = 0u;
  }
  __threadfence_system();
}

// One word per thread and round; a row's words stay together, so both sides are coalesced.
__global__ void __launch_bounds__(256) k_pack(uint32_t* __restrict__ dst, const char* __restrict__ src, size_t pitch, int w, int h) {
  for (int j = blockIdx.y; j < h; j += gridDim.y)
    for (int i = blockIdx.x * 256 + threadIdx.x; i < w; i += gridDim.x * 256)
      dst[(size_t)j * w + i] = __ldg(reinterpret_cast<const uint32_t*>(src + (size_t)j * pitch) + i);
}
void launch_pack(uint32_t* dst, const void* src, size_t pitch, int w, int h, cudaStream_t st) {
  if (w > 0 && h > 0)
    k_pack<<<dim3((w + 255) / 256, h < 2048 ? h : 2048), 256, 0, st>>>(dst, static_cast<const char*>(src), pitch, w, h);
}
void launch_write_params(uint32_t* dst, const ParamWords& b, int skip, int s0, int s1, cudaStream_t st) {
  k_write_params<<<1, 64, 0, st>>>(dst, b, skip, s0, s1);
}
void launch_write_pieces(float* dst, const PieceFloats& b, cudaStream_t st) {
  k_write_pieces<<<1, 256, 0, st>>>(dst, b);
}
void launch_readback(uint32_t* src, uint32_t* host, int nwords, int nzero, cudaStream_t st) {
  k_readback<<<1, 512, 0, st>>>(src, host, nwords, nzero);
}
void launch_project(SceneDesc* scenes, const Work* work, int ntiles, bool fp64, cudaStream_t st, int nscenes, int post,
                    const double* dxd, const double* alpha, float* dtv) {
  if (ntiles <= 0) return;
  if (fp64) k_project<true><<<ntiles, PR_TX * PR_TY, 0, st>>>(scenes, work, nscenes, post, dxd, alpha, dtv);
  else k_project<false><<<ntiles, PR_TX * PR_TY, 0, st>>>(scenes, work, nscenes, post, dxd, alpha, dtv);
}
void launch_cfl_update(SceneDesc* scenes, int nscenes, const double* dxd, const double* alpha, cudaStream_t st) {
  if (nscenes > 0) k_cfl_update<<<(nscenes + 127) / 128, 128, 0, st>>>(scenes, nscenes, dxd, alpha);
}
void launch_geometry(const SceneDesc* scenes, const Work* work, int ntiles, cudaStream_t st) {
  if (ntiles > 0) k_geometry<<<ntiles, GEO_TX * GEO_TY, 0, st>>>(scenes, work);
}
void launch_radiation(const SceneDesc* scenes, int scene, int nx, int ny, int ntargets, int nray, cudaStream_t st) {
  if (ntargets <= 0) return;
  k_emission<<<dim3((nx + 31) / 32, (ny + 7) / 8), 256, 0, st>>>(scenes, scene);
  // 16 rays per CTA spread few targets over the chip; from four such CTAs per SM on, 32 rays keep the
  // adding warp full. Both, whole pass: 160x224 with 16 pieces 25 and 31 us, 224x320 with 16 29 and
  // 37 us, 352x512 with 40 58 and 50 us.
  const int rt = (long)ntargets * nray > 4L * 148 * 16 ? 32 : 16;
  const int ncta = nray / rt < 1 ? 1 : nray / rt > RAD_CL ? RAD_CL : nray / rt;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ntargets * ncta);
  cfg.blockDim = dim3(RAD_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ncta; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (rt == 32) cudaLaunchKernelEx(&cfg, k_radiation<32>, scenes, scene, nray);
  else cudaLaunchKernelEx(&cfg, k_radiation<16>, scenes, scene, nray);
}
void launch_budgets(const SceneDesc* scenes, int scene, int cells, double* out, cudaStream_t st) {
  k_budgets<<<monitor_ctas(cells), 256, 0, st>>>(scenes, scene, out);
}

}  // namespace cfg
