// Fused multigrid V(2,2) cycle of shaders/pressure.wgsl (schedule of
// js/fluid.js:294-312) with temporal blocking.
//
// Each fine level l < lc is handled by two kernels per cycle:
//   down: stage p, rhs, ax, ay of the tile plus a 5-cell halo into shared
//         memory with TMA tensor copies, run the 4 colour passes (red, black,
//         red, black), each over the whole region and exact one cell further
//         in than the last, then the residual of the tile's cells and its
//         restriction to the coarse rhs (coarse p = 0);
//   up:   the same staging (and the coarse p under the tile), bilinear
//         prolongation of the coarse correction, 4 colour passes (black, red,
//         black, red); on level 0 also the residual norm (FP32 modes) or
//         p64 += p (FP64 defect correction).
// A cell update reads exactly the neighbour values the separate dispatches
// would read, so the result equals the reference schedule bit for bit.
// Down kernels read p and write pb; up kernels read pb and write p, so no CTA
// reads a halo another CTA is rewriting.
// Levels lc..coarsest run in one CTA per scene (coarse block): every level's
// arrays staged into shared memory by TMA bulk copies, __syncthreads between
// passes, and the coarsest level's 120 red-black sweeps (pressure.wgsl:132-156)
// in one warp's registers (levels that do not fit there: on one thread per
// red/black cell pair with a named barrier).
#include "gas_dev.cuh"
#include "kernels.h"
#include "reduce.cuh"
#include "mg_common.cuh"
#include "tma.cuh"

#include <algorithm>

namespace cfg {

namespace {

// Shared tile of the fused kernels: every array staged as an MGF_BW-wide box whose
// column 0 is level column sx and row 0 is level row sy (ay has one more row).
struct Tile {
  float *p, *rhs, *ax, *ay;
  int sx, sy;
  __device__ __forceinline__ int c(int i, int j) const { return (j - sy) * MGF_BW + (i - sx); }
};

// pressure.wgsl:77-85 on the shared tile (i, j in level coordinates); ax[c] is the
// west face of cell c, ay[c] its south face
__device__ __forceinline__ void stencil_s(const Tile& t, int nx, int ny, int i, int j, float& off, float& diag) {
  off = 0.f; diag = 0.f;
  const int k = t.c(i, j);
  const float w = t.ax[k], e = t.ax[k + 1], s = t.ay[k], n = t.ay[k + MGF_BW];
  if (i > 0) { off += w * t.p[k - 1]; diag += w; } else { diag += 2.f * w; }
  if (i < nx - 1) { off += e * t.p[k + 1]; diag += e; } else { diag += 2.f * e; }
  if (j > 0) { off += s * t.p[k - MGF_BW]; diag += s; }
  if (j < ny - 1) { off += n * t.p[k + MGF_BW]; diag += n; } else { diag += 2.f * n; }
}
// (L z)_ij in FP64 from the tile's f32 z and coefficients (pressure.wgsl:77-85 promoted,
// as the FP64 defect: (off - diag z) / h2, 0 in closed cells). The products of two f32 values
// are exact in FP64, so the fused multiply-adds round as the separate products and sums
// would; the division is a product with rh2 = 1 / h2 (FP64, one rounding more: the Krylov
// loop's own operator, the same in every kernel that forms it)
__device__ __forceinline__ double lap_tile64(const Tile& t, const LevelDesc& L, int i, int j, double rh2) {
  const int k = t.c(i, j);
  const double w = t.ax[k], e = t.ax[k + 1], s = t.ay[k], n = t.ay[k + MGF_BW];
  double off = 0.0, diag = 0.0;
  if (i > 0) { off = __fma_rn(w, (double)t.p[k - 1], off); diag += w; } else diag += 2.0 * w;
  if (i < L.nx - 1) { off = __fma_rn(e, (double)t.p[k + 1], off); diag += e; } else diag += 2.0 * e;
  if (j > 0) { off = __fma_rn(s, (double)t.p[k - MGF_BW], off); diag += s; }
  if (j < L.ny - 1) { off = __fma_rn(n, (double)t.p[k + MGF_BW], off); diag += n; } else diag += 2.0 * n;
  return diag > 0.0 ? __fma_rn(-diag, (double)t.p[k], off) * rh2 : 0.0;
}
__device__ __forceinline__ float diag_s(const Tile& t, int nx, int ny, int i, int j) {
  const int k = t.c(i, j);
  const float w = t.ax[k], e = t.ax[k + 1], s = t.ay[k], n = t.ay[k + MGF_BW];
  float diag = 0.f;
  if (i > 0) diag += w; else diag += 2.f * w;
  if (i < nx - 1) diag += e; else diag += 2.f * e;
  if (j > 0) diag += s;
  if (j < ny - 1) diag += n; else diag += 2.f * n;
  return diag;
}

constexpr uint32_t BOX_BYTES = MGF_BW * MGF_BH * 4, BOX_AY_BYTES = MGF_BW * (MGF_BH + 1) * 4;
constexpr uint32_t CBOX_BYTES = MGF_CBW * MGF_CBH * 4;

__device__ __forceinline__ const void* tmap_of(const SceneDesc& S, int level, int kind) {
  return S.tmap + (size_t)(level * TM_PER_LEVEL + kind) * TMAP_BYTES;
}

// Whether the scene has stopped cycling, asked before the wait on the previous kernel: the flag
// only falls during a loop (the kernels before the loop raise it, and no loop kernel starts
// before they have completed), so a zero stands whatever the previous kernel still does. A one
// may be stale; the flag is read again after the wait. A laid-out cycle after the last one
// needed then costs its kernels' launches only.
__device__ __forceinline__ bool scene_idle(const SolveState* ss) { return *(const volatile int*)&ss->active == 0; }

// Tile staging on two barriers around the wait on the previous kernel. stage_coef
// (before the wait in a one-scene engine, which also waits for them and builds the stencils
// before the wait, with the state copies' tensor maps prefetched; else after it, with
// stage_state, once the scene's flag says it still cycles): one thread initialises both barriers and requests the coefficients
// ax, ay on bar[0]; they are built before the pressure loop and written by no loop kernel
// (the first cycle's first kernel starts once the kernels that build them have completed: it is
// launched without programmatic dependence, or is a loop body's first node). stage_state
// (after the wait): p from map `pkind`, rhs and the coarse p under the tile on bar[1]; with
// `copy` false nothing is requested and bar[1] completes on its arrival; with `pload` false p
// is not copied (the caller zero-fills its box). With one scene the copies are issued before
// its `active` flag is read again, which then overlaps them; with several once the flag says
// that the scene cycles. tile_wait: all threads wait for one barrier (bounded); false in every thread if a
// wait ran out, after recording the error and waiting once more for the copies in flight.
__device__ __forceinline__ void stage_coef(const SceneDesc& S, int level, const Tile& t, uint64_t* bar) {
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_arrive_expect_tx(&bar[0], BOX_BYTES + BOX_AY_BYTES);
    tma_load_2d(t.ax, tmap_of(S, level, TM_AX), t.sx, t.sy, &bar[0]);
    tma_load_2d(t.ay, tmap_of(S, level, TM_AY), t.sx, t.sy, &bar[0]);
  }
}
// the tensor maps of stage_state's copies (coef: and of stage_coef's) into the descriptor cache
// (before the wait)
__device__ __forceinline__ void prefetch_state_maps(const SceneDesc& S, int level, int pkind, bool coarse, bool coef = false) {
  if (threadIdx.x == 0) {
    if (coef) { tmap_prefetch(tmap_of(S, level, TM_AX)); tmap_prefetch(tmap_of(S, level, TM_AY)); }
    tmap_prefetch(tmap_of(S, level, pkind));
    tmap_prefetch(tmap_of(S, level, TM_RHS));
    if (coarse) tmap_prefetch(tmap_of(S, level + 1, TM_PC));
  }
}
__device__ __forceinline__ void stage_state(const SceneDesc& S, int level, int pkind, const Tile& t, bool copy,
                                            float* cp, int cx, int cy, uint64_t* bar, bool pload = true) {
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(&bar[1], copy ? (pload ? 2 : 1) * BOX_BYTES + (cp ? CBOX_BYTES : 0u) : 0u);
    if (copy) {
      if (pload) tma_load_2d(t.p, tmap_of(S, level, pkind), t.sx, t.sy, &bar[1]);
      tma_load_2d(t.rhs, tmap_of(S, level, TM_RHS), t.sx, t.sy, &bar[1]);
      if (cp) tma_load_2d(cp, tmap_of(S, level + 1, TM_PC), cx, cy, &bar[1]);
    }
  }
}
__device__ __forceinline__ bool tile_wait(uint64_t* bar, SolveCtl* ctl) {
  const bool ok = mbar_wait(bar, 0);
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) atomicExch(&ctl->err, 1);
    mbar_wait(bar, 0);
    return false;
  }
  return true;
}
// both barriers of a tile: the coefficients (then `between`, e.g. the stencils), the state
template <class F>
__device__ __forceinline__ bool tile_wait2(uint64_t* bar, SolveCtl* ctl, F&& between) {
  if (!tile_wait(&bar[0], ctl)) {
    mbar_wait(&bar[1], 0);
    return false;
  }
  between();
  return tile_wait(&bar[1], ctl);
}


// ---- packed pairs of f32: one instruction for two operations, each rounded as its scalar form.
// A product is the fused multiply-add with -0 (a b + -0 rounds to a b, signs of zero kept), its -0
// an argument of the kernel: the assembler contracts mul.rn.f32x2 with an add.rn.f32x2 that
// follows it, whatever -fmad says, and a fused one with a -0 that it can see as well.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f2 lds2(const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return pk(v.x, v.y); }
__device__ __forceinline__ void sts2(float* p, f2 v) { float2 w; upk(v, w.x, w.y); *reinterpret_cast<float2*>(p) = w; }

// The four colour passes of a fused kernel. Thread t owns item t of pass 1's region (40 x 24 cells,
// 240 items): the four cells (base..base+3, j) of one row, base even, which are two cells of each
// colour. Their stencils stay in registers as packed pairs by colour, and so do the cells' own
// values. The tile's p is held twice 26 columns to a row, red cells and black ones apart (column
// pair c of box row r: sp[r SPW + c] and sp[r SPW + SPB + c]): a pass then reads the other colour
// of the rows below and above as one aligned pair each and one neighbour beside the item; the
// rest of the row is the item's own. Passes 2-4 update the whole region again: a cell at distance d from its
// edge is exact through pass d, a later update there only spoils values that no cell
// needed later reads (pass k of a cell at distance >= k reads cells at distance >= k - 1). Cells
// outside the level and closed ones have zeros throughout and stay zero. The sums leave out
// the leading +0 of pressure.wgsl:77-85, which changes no value. The quotient is div_by_rcp's.
constexpr int RG_W = MGF_TX + 2 * MGF_H - 2, RG_H = MGF_TY + 2 * MGF_H - 2;   // pass 1's region
constexpr int RG_IW = RG_W / 4, RG_N = RG_IW * RG_H;                          // items per row, items
static_assert(RG_W % 4 == 0 && RG_N <= 256 && MGF_H == 5 && MGF_SX == 8, "one item per thread");
constexpr int SPB = 26, SPW = 2 * SPB, SP_N = MGF_BH * SPW;   // 52 words per row: pairs of 3 rows hit 32 banks evenly
struct Item {
  int r, j, base, k, c;   // region row, level row, first cell's level column, box index, column pair
  bool on, odd;           // owns an item; j odd: the red cells are base+1, base+3
};
__device__ __forceinline__ Item item_of(int x0, int y0) {
  Item q;
  q.on = threadIdx.x < RG_N;
  q.r = threadIdx.x / RG_IW;
  const int a = threadIdx.x - q.r * RG_IW;
  q.j = y0 - MGF_H + 1 + q.r;
  q.base = x0 - MGF_H + 1 + 4 * a;
  q.k = (q.r + 1) * MGF_BW + MGF_SX - MGF_H + 1 + 4 * a;
  q.c = (MGF_SX - MGF_H + 1) / 2 + 2 * a;
  q.odd = q.j & 1;
  return q;
}
// whether the item lies in the tile
__device__ __forceinline__ bool in_tile(const Item& q, int x0, int y0) {
  return q.on && q.base >= x0 && q.base < x0 + MGF_TX && q.j >= y0 && q.j < y0 + MGF_TY;
}
// four values in column order as pairs by colour, and back
__device__ __forceinline__ void by_colour(const Item& q, const float (&v)[4], f2 (&c)[2]) {
  const f2 e = pk(v[0], v[2]), o = pk(v[1], v[3]);
  c[0] = q.odd ? o : e; c[1] = q.odd ? e : o;
}
__device__ __forceinline__ float4 in_order(const Item& q, const f2 (&c)[2]) {
  float4 v;
  upk(q.odd ? c[1] : c[0], v.x, v.z);
  upk(q.odd ? c[0] : c[1], v.y, v.w);
  return v;
}
struct Sten { f2 w[2], e[2], s[2], n[2], nd[2], rc[2], nrh[2], nz; };   // nd: -diag, rc: RN(1/diag), nrh: -(rhs h2), nz: -0
// the stencils from the coefficients alone
__device__ __forceinline__ void item_stencils(const Tile& t, const LevelDesc& L, const Item& q, Sten& c) {
  float w[4], e[4], s[4], n[4], nd[4], rc[4];
  #pragma unroll
  for (int m = 0; m < 4; m++) w[m] = e[m] = s[m] = n[m] = nd[m] = rc[m] = 0.f;
  if (q.on && (unsigned)q.j < (unsigned)L.ny) {
    const float4 A = *reinterpret_cast<const float4*>(t.ax + q.k), Sv = *reinterpret_cast<const float4*>(t.ay + q.k),
                 Nv = *reinterpret_cast<const float4*>(t.ay + q.k + MGF_BW);
    const float a[5] = {A.x, A.y, A.z, A.w, t.ax[q.k + 4]}, sv[4] = {Sv.x, Sv.y, Sv.z, Sv.w}, nv[4] = {Nv.x, Nv.y, Nv.z, Nv.w};
    #pragma unroll
    for (int m = 0; m < 4; m++) {
      const int i = q.base + m;
      float d = i > 0 ? a[m] : 2.f * a[m];
      d += i < L.nx - 1 ? a[m + 1] : 2.f * a[m + 1];
      if (q.j > 0) d += sv[m];
      d += q.j < L.ny - 1 ? nv[m] : 2.f * nv[m];
      if ((unsigned)i < (unsigned)L.nx && d > 0.f) {
        w[m] = a[m]; e[m] = a[m + 1]; s[m] = sv[m]; n[m] = nv[m]; nd[m] = -d; rc[m] = __frcp_rn(d);
      }
    }
  }
  by_colour(q, w, c.w); by_colour(q, e, c.e); by_colour(q, s, c.s); by_colour(q, n, c.n);
  by_colour(q, nd, c.nd); by_colour(q, rc, c.rc);
}
// the item's rhs (column order) into the stencils; kept apart for the residual where `rhs` asks
__device__ __forceinline__ void item_rhs(const Item& q, float h2, const float4 r, Sten& c, f2* rhs = nullptr) {
  const float v[4] = {r.x, r.y, r.z, r.w};
  f2 x[2];
  by_colour(q, v, x);
  const f2 m = pk(-h2, -h2);
  c.nrh[0] = mul2(x[0], m, c.nz); c.nrh[1] = mul2(x[1], m, c.nz);
  if (rhs) { rhs[0] = x[0]; rhs[1] = x[1]; }
}
// the sum of coefficient times neighbour for the item's cells of colour col, in the reference's
// order (west, east, south, north); own: the item's cells of the other colour
__device__ __forceinline__ f2 item_off(const float* sp, const Item& q, const Sten& c, int col, f2 own) {
  const float* o = sp + (q.r + 1) * SPW + (1 - col) * SPB + q.c;   // the other colour's row
  const bool hi = q.odd != (col == 1);   // this colour's cells are base+1, base+3
  float o0, o1;
  upk(own, o0, o1);
  const float x = o[hi ? 2 : -1], y = hi ? o1 : o0;
  f2 off = mul2(c.w[col], pk(hi ? o0 : x, y), c.nz);
  off = add2(off, mul2(c.e[col], pk(y, hi ? x : o1), c.nz));
  off = add2(off, mul2(c.s[col], lds2(o - SPW), c.nz));
  off = add2(off, mul2(c.n[col], lds2(o + SPW), c.nz));
  return off;
}
__device__ __forceinline__ f2 quot2(f2 x, f2 nd, f2 r, f2 nz) {   // div_by_rcp; nd: minus the divisor
  const f2 q0 = mul2(x, r, nz);
  return fma2(fma2(q0, nd, x), r, q0);
}
// p[col]: the item's own values, also in sp; on return the smoothed ones
__device__ __forceinline__ void item_passes(float* sp, const Item& q, const Sten& c, int first, f2 (&p)[2]) {
  #pragma unroll
  for (int k = 0; k < 4; k++) {
    const int col = (first + k) & 1;
    if (q.on) {
      p[col] = quot2(add2(item_off(sp, q, c, col, p[1 - col]), c.nrh[col]), c.nd[col], c.rc[col], c.nz);
      sts2(sp + (q.r + 1) * SPW + col * SPB + q.c, p[col]);
    }
    __syncthreads();
  }
}
__device__ __forceinline__ void put_item(float* sp, const Item& q, const f2 (&p)[2]) {
  sts2(sp + (q.r + 1) * SPW + q.c, p[0]);
  sts2(sp + (q.r + 1) * SPW + SPB + q.c, p[1]);
}
// The ring of one cell about pass 1's region, whose values pass 1 reads: ring cell e's box row and
// column (two rows of 42, then two columns of 24)
constexpr int RING_N = 2 * (RG_W + 2) + 2 * RG_H;
static_assert(RING_N <= 256, "one ring cell per thread");
__device__ __forceinline__ void ring_cell(int e, int& br, int& bc) {
  constexpr int w = RG_W + 2;
  if (e < 2 * w) { br = e < w ? 0 : RG_H + 1; bc = MGF_SX - MGF_H + (e < w ? e : e - w); }
  else { e -= 2 * w; br = 1 + (e >> 1); bc = MGF_SX - MGF_H + ((e & 1) ? RG_W + 1 : 0); }
}
// where box cell (br, bc) of the tile at (sx, sy) lies in sp
__device__ __forceinline__ int sp_at(int br, int bc, int sx, int sy) {
  return br * SPW + (((sx + bc + sy + br) & 1) ? SPB : 0) + (bc >> 1);
}
// p of the box into sp as it is (level 0 from a start that is not zero), or zeros
__device__ __forceinline__ void stage_sp(const Tile& t, float* sp, const Item& q, f2 (&p)[2]) {
  if (q.on) {
    const float4 v = *reinterpret_cast<const float4*>(t.p + q.k);
    const float a[4] = {v.x, v.y, v.z, v.w};
    by_colour(q, a, p);
    put_item(sp, q, p);
  }
  if (threadIdx.x < RING_N) {
    int br, bc;
    ring_cell(threadIdx.x, br, bc);
    sp[sp_at(br, bc, t.sx, t.sy)] = t.p[br * MGF_BW + bc];
  }
}
__device__ __forceinline__ void zero_sp(float* sp, f2 (&p)[2]) {
  for (int e = threadIdx.x; e < SP_N / 4; e += 256) reinterpret_cast<float4*>(sp)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  p[0] = p[1] = 0ull;
}
static_assert(SP_N % 4 == 0, "filled by float4");

// The up kernel's prolongation (pressure.wgsl:116-129) over the region and its ring: the bilinear
// correction from the coarse box at (cx, cy), added to open cells. An item's four cells lie over two
// coarse cells; its sums are formed as packed pairs (cells 0, 1 and 2, 3).
__device__ __forceinline__ void prolong_item(const Tile& t, const LevelDesc& C, const Item& q, const Sten& c, int cx, int cy,
                                             const float* scp, f2 (&p)[2]) {
  const int I = q.base / 2, J = q.j / 2;
  const int J2 = min(max(J + ((q.j & 1) ? 1 : -1), 0), C.ny - 1);
  const int il = max(I - 1, 0), ir = min(I + 2, C.nx - 1), im = min(I + 1, C.nx - 1);
  const float* a = scp + (J - cy) * MGF_CBW - cx;
  const float* b = scp + (J2 - cy) * MGF_CBW - cx;
  const float a0 = a[I], a1 = a[im], al = a[il], ar = a[ir], b0 = b[I], b1 = b[im], bl = b[il], br = b[ir];
  const f2 k0 = pk(0.5625f, 0.5625f), k1 = pk(0.1875f, 0.1875f), k2 = pk(0.0625f, 0.0625f);
  const f2 z = c.nz;
  f2 u = add2(add2(mul2(k0, pk(a0, a0), z), mul2(k1, add2(pk(al, a1), pk(b0, b0)), z)), mul2(k2, pk(bl, b1), z));
  f2 v = add2(add2(mul2(k0, pk(a1, a1), z), mul2(k1, add2(pk(a0, ar), pk(b1, b1)), z)), mul2(k2, pk(b0, br), z));
  float x[4];
  upk(u, x[0], x[1]);
  upk(v, x[2], x[3]);
  f2 d[2];
  by_colour(q, x, d);
  // closed cells and cells outside the level (zero diagonal) add nothing
  #pragma unroll
  for (int col = 0; col < 2; col++) {
    float r0, r1, x0, x1;
    upk(c.rc[col], r0, r1);
    upk(d[col], x0, x1);
    d[col] = pk(r0 != 0.f ? x0 : 0.f, r1 != 0.f ? x1 : 0.f);
  }
  const float4 f = *reinterpret_cast<const float4*>(t.p + q.k);
  const float y[4] = {f.x, f.y, f.z, f.w};
  by_colour(q, y, p);
  p[0] = add2(p[0], d[0]); p[1] = add2(p[1], d[1]);
}
// a ring cell's plan, from the coefficients and level sizes alone: bits 0-10 box index, 11-19 its
// coarse cell in the coarse box, 20-21 and 22-23 the steps to the other coarse column and row plus
// one, 24 open
static_assert(MGF_BW * MGF_BH <= 2048 && MGF_CBW * MGF_CBH <= 512, "plan fields");
__device__ __forceinline__ uint32_t ring_plan(const Tile& t, const LevelDesc& L, const LevelDesc& C, int cx, int cy) {
  if (threadIdx.x >= RING_N) return 0u;
  int br, bc;
  ring_cell(threadIdx.x, br, bc);
  const int i = t.sx + bc, j = t.sy + br;
  const uint32_t k = br * MGF_BW + bc;
  if (i < 0 || i >= L.nx || j < 0 || j >= L.ny) return k;
  const int I = i / 2, J = j / 2;
  const int dI = min(max(I + ((i & 1) == 1 ? 1 : -1), 0), C.nx - 1) - I;
  const int dJ = min(max(J + ((j & 1) == 1 ? 1 : -1), 0), C.ny - 1) - J;
  return k | (uint32_t)((J - cy) * MGF_CBW + I - cx) << 11 | (uint32_t)(dI + 1) << 20 | (uint32_t)(dJ + 1) << 22 |
         (diag_s(t, L.nx, L.ny, i, j) > 0.f ? 1u << 24 : 0u);
}
__device__ __forceinline__ void prolong_ring(const Tile& t, float* sp, const float* scp, uint32_t pl) {
  if (threadIdx.x >= RING_N) return;
  const int k = pl & 2047, br = k / MGF_BW, bc = k - br * MGF_BW;
  float c = 0.f;
  if (pl & (1u << 24)) {
    const int a = (pl >> 11) & 511, dI = (int)((pl >> 20) & 3) - 1, dJ = ((int)((pl >> 22) & 3) - 1) * MGF_CBW;
    c = 0.5625f * scp[a] + 0.1875f * (scp[a + dI] + scp[a + dJ]) + 0.0625f * scp[a + dI + dJ];
  }
  sp[sp_at(br, bc, t.sx, t.sy)] = t.p[k] + c;
}
// four values of a level row from column i on (those inside the level)
__device__ __forceinline__ void store4(float* row, int i, int nx, float4 v) {
  if (i + 3 < nx) { *reinterpret_cast<float4*>(row + i) = v; return; }
  if (i < nx) row[i] = v.x;
  if (i + 1 < nx) row[i + 1] = v.y;
  if (i + 2 < nx) row[i + 2] = v.z;
}

// Fused Krylov mode on level 0 (all scenes' coarse blocks start below it). The update of
// cycle c (d = z + beta d, q = Lz + beta q, p64 += alpha d, r -= alpha q with cycle c's
// alpha, beta) is split: the next cycle's down kernel forms d and p64 on its tile and the
// new rhs0 = f32(r - alpha q) on pass 1's region from the stored r, q, Lz (read only
// there, so no CTA reads a value another rewrites); the next up kernel rewrites r and q on
// its tile before its dot products; the update of the last cycle is applied by
// k_pcg_finish after the loop. The up kernel's tiles leave their nine dot products as
// partials; k_pcg_decide (one CTA per scene, the next kernel) sums them, forms the cycle's
// alpha and beta, and ||r_c||^2 = r.r - 2 alpha r.q_c + alpha^2 q_c.q_c (q_c = Lz + beta q)
// for the loop decision.
// Two consecutive doubles of a dense FP64 row (nx is even on a level with one below it, and the
// column too: 16-byte aligned)
__device__ __forceinline__ double2 ldcg2(const double* p) { return __ldcg(reinterpret_cast<const double2*>(p)); }
// the item's new rhs0 in column order, from its stored r, q, Lz
__device__ __forceinline__ float4 pcg_rhs(const SceneDesc& S, const LevelDesc& L, const Item& q, const PcgPrev& pv) {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (q.on && (unsigned)q.j < (unsigned)L.ny) {
    const bool first = pv.cycles == 1;
    #pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = q.base + 2 * h;
      if (i < 0 || i >= L.nx) continue;
      const size_t k = (size_t)q.j * L.nx + i;
      const double2 r = ldcg2(S.r64 + k), qq = ldcg2(S.q64 + k), lz = ldcg2(S.dB + k);
      v[2 * h] = (float)(r.x - pv.alpha * (first ? lz.x : lz.x + pv.beta * qq.x));
      v[2 * h + 1] = (float)(r.y - pv.alpha * (first ? lz.y : lz.y + pv.beta * qq.y));
    }
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}
// d and p64 of the item's cells (z: the last cycle's p)
__device__ __forceinline__ void pcg_dir(const SceneDesc& S, const LevelDesc& L, const Item& q, const PcgPrev& pv) {
  if (q.j >= L.ny) return;
  const bool first = pv.cycles == 1;
  #pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = q.base + 2 * h;
    if (i >= L.nx) continue;
    const size_t k = (size_t)q.j * L.nx + i;
    const float2 z = __ldcg(reinterpret_cast<const float2*>(L.p + (size_t)q.j * L.pc + i));
    double2 d = ldcg2(S.dA + k), p = ldcg2(S.p64 + k);
    d.x = first ? (double)z.x : (double)z.x + pv.beta * d.x;
    d.y = first ? (double)z.y : (double)z.y + pv.beta * d.y;
    p.x += pv.alpha * d.x;
    p.y += pv.alpha * d.y;
    *reinterpret_cast<double2*>(S.dA + k) = d;
    *reinterpret_cast<double2*>(S.p64 + k) = p;
  }
}

}  // namespace

// ------------------------------------------------------------------ down: 4 passes + restrict
// PCG: the fused Krylov update on level 0 (above)
// ONE: compiled for an engine of one scene (nscenes == 1), whose flag only ends the loop
// MINB: resident CTAs per SM the registers are sized for: three for one scene (four cost 512x768
// 3.5% per step), two for its level-0 Krylov kernels where the tiles fit in one wave at two per SM
// (256x384: three cost 2%), four for several scenes (64 uneven ones: three cost 5%, five 7%)
// Bound by instruction issue where the tiles fill the GPU and by the chain copy - passes - stores
// where they do not. With each thread's two cells of each colour a stride apart and unpacked
// arithmetic (scalar loads of four neighbours and four coefficients per cell, the FP64 update and
// the stencils in different maps) a step took 814 us at 512x768, 288 at 256x384, 95.4 at 224x320
// and 4655 for the 64-scene batch; with items 741, 270, 91.9 and 3903.
template <int TX, int TY, bool PCG, bool ONE, int MINB = ONE ? 3 : 4>
__global__ void __launch_bounds__(256, MINB) k_mg_down(const SceneDesc* __restrict__ scenes, int nscenes, const Work* __restrict__ work,
                                                 int level, SolveCtl* ctl, int count_iter, f2 nz) {
  static_assert(TX == MGF_TX && TY == MGF_TY, "the tensor-map boxes are built for the MGF tile");
  __shared__ __align__(128) float bp[MGF_BH * MGF_BW];
  __shared__ __align__(128) float srhs[MGF_BH * MGF_BW];
  __shared__ __align__(128) float sax[MGF_BH * MGF_BW];
  __shared__ __align__(128) float say[(MGF_BH + 1) * MGF_BW];
  __shared__ __align__(16) float sp[SP_N];
  __shared__ __align__(16) float sr[TY / 2 * TX];   // odd rows' residuals
  __shared__ __align__(8) uint64_t bar[2];
  const Work w = work[blockIdx.x];
  const SceneDesc& S = scenes[w.scene];
  pdl_trigger();
  const LevelDesc L = S.lev[level], C = S.lev[level + 1];
  const int x0 = w.tx * TX, y0 = w.ty * TY;
  const Tile t{bp, srhs, sax, say, x0 - MGF_SX, y0 - MGF_H};
  const Item q = item_of(x0, y0);
  const bool on = S.enabled;   // host-written, constant during the step
  SolveState* ss = S.solve;
  // one scene: its flag only ends the loop, so the tile is requested before it is read;
  // several: a scene that stopped loads nothing
  constexpr bool spec = ONE;
  __shared__ int s_idle;   // thread 0's reading: the flag may fall while the CTA's threads would read it
  if (on && spec && threadIdx.x == 0) {
    const bool z = scene_idle(ss);
    s_idle = z;
    if (!z) {
      stage_coef(S, level, t, bar);
      prefetch_state_maps(S, level, TM_P, false);
    }
  }
  // below level 0 the level's p is zero on entry (the restriction above zeroes it)
  const bool pz = level > 0;
  // several scenes: mostly more tiles than fit at once, so nothing is gained before the wait; what the
  // copies depend on is read in one round, and all of them are requested together, their tensor maps
  // prefetched (64 uneven scenes: 3878 -> 3826 us per step)
  PcgPrev pv{};
  bool live = true;
  if (!spec) {
    prefetch_state_maps(S, level, TM_P, false, true);
    pdl_wait();
    if (on) {
      live = *(volatile int*)&ss->active != 0;
      if (PCG) pv = pcg_load(ss);
    }
  }
  f2 p[2];
  zero_sp(sp, p);
  if (!spec && on && live && threadIdx.x == 0) {
    stage_coef(S, level, t, bar);
    stage_state(S, level, TM_P, t, !(PCG && pv.cycles >= 1), nullptr, 0, 0, bar, !pz);
  }
  __syncthreads();
  const bool idle = on && spec && s_idle;
  // one scene: the stencils, which depend on the coefficients alone, are built before the wait
  Sten c;
  c.nz = nz;
  bool ok = true;
  if (on && spec && !idle && (ok = tile_wait(&bar[0], ctl))) item_stencils(t, L, q, c);
  if (spec) pdl_wait();
  if (count_iter && blockIdx.x == 0 && threadIdx.x == 0) loop_count(ctl);
  if (!on || !ok || idle) return;
  if (spec) {
    if (PCG) pv = pcg_load(ss);
    live = *(volatile int*)&ss->active != 0;
  } else if (!live) {
    return;
  }
  const bool upd = PCG && pv.cycles >= 1;   // an update of the previous cycle is pending
  if (spec) stage_state(S, level, TM_P, t, !upd, nullptr, 0, 0, bar, !pz);
  float4 rv = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool mine = in_tile(q, x0, y0);
  if (PCG && upd && live) {
    rv = pcg_rhs(S, L, q, pv);
    // the pending direction and pressure (read and written by this item alone): with several scenes beside
    // the copies, with one after the results that the next kernel waits for
    if (!spec && mine) pcg_dir(S, L, q, pv);
  }
  if (!(spec ? tile_wait(&bar[1], ctl) : tile_wait2(bar, ctl, [&] { item_stencils(t, L, q, c); })) || !live)
    return;
  f2 rhs[2];
  if (upd) {
    // rhs0 of the tile also to global, for the up kernel's staging
    if (mine && q.j < L.ny) store4(L.rhs + (size_t)q.j * L.pc, q.base, L.nx, rv);
  } else if (q.on) {
    rv = *reinterpret_cast<const float4*>(t.rhs + q.k);
  }
  item_rhs(q, L.h2, rv, c, rhs);
  if (!upd && !pz) {
    stage_sp(t, sp, q, p);
    __syncthreads();
  }
  item_passes(sp, q, c, 0, p);   // colours 0, 1, 0, 1 (js/fluid.js:298-301)
  // residual of the tile cells (pressure.wgsl:96-101) from the items' stencils; the quotient by h2
  // from RN(1/h2), the IEEE one; then the restriction (pressure.wgsl:104-113): the even rows' items
  // add the odd rows' residuals to their own
  float4 res = make_float4(0.f, 0.f, 0.f, 0.f);
  const int tr = q.r - (MGF_H - 1), ti = q.base - x0;   // tile row and column
  if (mine) {
    const float h = L.h2, rh = __frcp_rn(h);
    const f2 nh = pk(-h, -h), rh2 = pk(rh, rh), m1 = pk(-1.f, -1.f);
    f2 r[2];
    #pragma unroll
    for (int col = 0; col < 2; col++) {
      const f2 x = add2(item_off(sp, q, c, col, p[1 - col]), mul2(c.nd[col], p[col], c.nz));
      r[col] = fma2(quot2(x, nh, rh2, c.nz), m1, rhs[col]);
      float r0, r1, d0, d1;
      upk(c.rc[col], d0, d1);
      upk(r[col], r0, r1);
      r[col] = pk(d0 != 0.f ? r0 : 0.f, d1 != 0.f ? r1 : 0.f);
    }
    res = in_order(q, r);
    if (tr & 1) *reinterpret_cast<float4*>(sr + (tr >> 1) * TX + ti) = res;
    if (q.j < L.ny) store4(L.pb + (size_t)q.j * L.pc, q.base, L.nx, in_order(q, p));   // the smoothed p
  }
  __syncthreads();
  if (mine && !(tr & 1)) {
    const float4 o = *reinterpret_cast<const float4*>(sr + (tr >> 1) * TX + ti);
    const int I = q.base / 2, J = q.j / 2;
    if (J < C.ny) {
      const float v0 = 0.25f * (res.x + res.y + o.x + o.y), v1 = 0.25f * (res.z + res.w + o.z + o.w);
      float* cr = C.rhs + (size_t)J * C.pc + I;
      float* cp = C.p + (size_t)J * C.pc + I;
      if (I + 1 < C.nx) {
        *reinterpret_cast<float2*>(cr) = make_float2(v0, v1);
        *reinterpret_cast<float2*>(cp) = make_float2(0.f, 0.f);
      } else if (I < C.nx) {
        *cr = v0;
        *cp = 0.f;
      }
    }
  }
  if (PCG && spec && upd && mine) pcg_dir(S, L, q, pv);
}

// ------------------------------------------------------------------ up: prolong + 4 passes (+ level-0 tail)
// tail: 0 none, 1 residual norm + loop decision (FP32 modes), 2 p64 += p (FP64 defect correction),
// 3 r.z, q.z, z.Lz -> the direction update (Krylov FP64 mode), 4 the same in the fused Krylov
// mode (the pending r, q update first; the loop decision from the recurrence for ||r||); one
// instance per tail (levels below 0: tail 0)
template <int TX, int TY, int TAIL, bool ONE, int MINB = ONE ? 3 : 4>   // ONE, MINB: as in k_mg_down
__global__ void __launch_bounds__(256, MINB) k_mg_up(const SceneDesc* __restrict__ scenes, int nscenes, const Work* __restrict__ work,
                                               int level, SolveCtl* ctl, f2 nz) {
  static_assert(TX == MGF_TX && TY == MGF_TY, "the tensor-map boxes are built for the MGF tile");
  static_assert(TAIL >= 0 && TAIL <= 4, "tails 0-4");
  constexpr bool KRY = TAIL == 4;
  constexpr int tail = TAIL;
  __shared__ __align__(128) float bp[MGF_BH * MGF_BW];
  __shared__ __align__(128) float srhs[MGF_BH * MGF_BW];
  __shared__ __align__(128) float sax[MGF_BH * MGF_BW];
  __shared__ __align__(128) float say[(MGF_BH + 1) * MGF_BW];
  __shared__ __align__(128) float scp[MGF_CBH * MGF_CBW];
  __shared__ __align__(16) float sp[SP_N];
  __shared__ double red[32];
  __shared__ __align__(8) uint64_t bar[2];
  const Work w = work[blockIdx.x];
  const SceneDesc& S = scenes[w.scene];
  pdl_trigger();
  const LevelDesc L = S.lev[level], C = S.lev[level + 1];
  const int x0 = w.tx * TX, y0 = w.ty * TY;
  const Tile t{bp, srhs, sax, say, x0 - MGF_SX, y0 - MGF_H};
  const Item q = item_of(x0, y0);
  // coarse p under the region: columns x0/2-4 .. x0/2+TX/2+3, rows y0/2-4 .. y0/2+TY/2+3
  const int cx = x0 / 2 - 8, cy = y0 / 2 - 4;
  const bool on = S.enabled;   // host-written, constant during the step
  SolveState* ss = S.solve;
  constexpr bool spec = ONE;   // as in k_mg_down
  PcgPrev pv{};
  bool live = true;
  if (!spec) {
    prefetch_state_maps(S, level, TM_PB, true, true);
    pdl_wait();
    if (on) {
      live = *(volatile int*)&ss->active != 0;
      if (KRY) pv = pcg_load(ss);
      if (live && threadIdx.x == 0) {
        stage_coef(S, level, t, bar);
        stage_state(S, level, TM_PB, t, true, scp, cx, cy, bar);
      }
    }
  }
  __shared__ int s_idle;
  if (on && spec && threadIdx.x == 0) {
    const bool z = scene_idle(ss);
    s_idle = z;
    if (!z) {
      stage_coef(S, level, t, bar);
      prefetch_state_maps(S, level, TM_PB, true);
    }
  }
  __shared__ double s_rh2;   // the FP64 operator's 1 / h2 (tails 3 and 4)
  if ((tail == 3 || tail == 4) && threadIdx.x == 0) s_rh2 = 1.0 / (double)L.h2;
  __syncthreads();
  const bool idle = on && spec && s_idle;
  const double rh2 = tail == 3 || tail == 4 ? s_rh2 : 0.0;
  Sten c;
  c.nz = nz;
  uint32_t pl = 0u;
  bool ok = true;
  auto prepare = [&] {
    item_stencils(t, L, q, c);
    pl = ring_plan(t, L, C, cx, cy);
  };
  if (on && spec && !idle && (ok = tile_wait(&bar[0], ctl))) prepare();
  if (spec) pdl_wait();
  if (!on || !ok || idle) return;
  if (spec) {
    stage_state(S, level, TM_PB, t, true, scp, cx, cy, bar);
    live = *(volatile int*)&ss->active != 0;
  } else if (!live) {
    return;
  }
  // fused Krylov mode: the solve state and this thread's stored r, q, Lz, read beside the copies
  double r0[2] = {0.0, 0.0}, q0[2] = {0.0, 0.0}, lz0[2] = {0.0, 0.0};
  if (KRY) {
    if (spec) pv = pcg_load(ss);
    #pragma unroll
    for (int m = 0; m < 2; m++) {
      const int e = threadIdx.x + 256 * m;
      const int i = x0 + e % TX, j = y0 + e / TX;
      if (i < L.nx && j < L.ny) {
        const int kk = j * L.nx + i;
        r0[m] = __ldcg(S.r64 + kk); q0[m] = __ldcg(S.q64 + kk); lz0[m] = __ldcg(S.dB + kk);
      }
    }
  }
  if (!(spec ? tile_wait(&bar[1], ctl) : tile_wait2(bar, ctl, prepare)) || !live)
    return;
  // prolongation (pressure.wgsl:116-129) on the whole region
  f2 p[2] = {0ull, 0ull};
  if (q.on) {
    item_rhs(q, L.h2, *reinterpret_cast<const float4*>(t.rhs + q.k), c);
    prolong_item(t, C, q, c, cx, cy, scp, p);
    put_item(sp, q, p);
  }
  prolong_ring(t, sp, scp, pl);
  __syncthreads();
  item_passes(sp, q, c, 1, p);   // colours 1, 0, 1, 0 (js/fluid.js:307-310)
  if (in_tile(q, x0, y0) && q.j < L.ny) store4(L.p + (size_t)q.j * L.pc, q.base, L.nx, in_order(q, p));
  if (tail == 0) return;
  // the tails read the tile and its ring from the box again
  if (q.on) *reinterpret_cast<float4*>(t.p + q.k) = in_order(q, p);
  __syncthreads();
  if (KRY) {
    // the pending r, q update (cycles >= 1), then r.z, q.z, z.Lz and the recurrence's r.r,
    // r.Lz, r.q, Lz.Lz, Lz.q, q.q on the tile
    const bool upd = pv.cycles >= 1, first = pv.cycles == 1;
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    #pragma unroll
    for (int m = 0; m < 2; m++) {
      const int e = threadIdx.x + 256 * m;
      const int i = x0 + e % TX, j = y0 + e / TX;
      if (i >= L.nx || j >= L.ny) continue;
      const int k = t.c(i, j), kk = j * L.nx + i;
      double r = r0[m], qv = q0[m];
      if (upd) {
        qv = first ? lz0[m] : lz0[m] + pv.beta * qv;
        r = r - pv.alpha * qv;
        S.q64[kk] = qv;
        S.r64[kk] = r;
      }
      const double z = (double)t.p[k];
      const double lz = lap_tile64(t, L, i, j, rh2);
      S.dB[kk] = lz;
      v[0] = __fma_rn(r, z, v[0]); v[1] = __fma_rn(qv, z, v[1]); v[2] = __fma_rn(z, lz, v[2]);
      v[3] = __fma_rn(r, r, v[3]); v[4] = __fma_rn(r, lz, v[4]); v[5] = __fma_rn(r, qv, v[5]);
      v[6] = __fma_rn(lz, lz, v[6]); v[7] = __fma_rn(lz, qv, v[7]); v[8] = __fma_rn(qv, qv, v[8]);
    }
    // the tile's nine partials, quantity-major (part[m * nt_up0 + tile]); k_pcg_decide sums
    // them once this kernel has completed (no arrival, no fence in these CTAs)
    __shared__ double redt[9 * 256 + 9];
    block_sum_t<9>(v, redt);
    if (threadIdx.x == 0)
      #pragma unroll
      for (int m = 0; m < 9; m++) S.part[m * S.nt_up0 + w.tile] = v[m];
    return;
  }
  double part = 0.0, part2 = 0.0, part3 = 0.0;
  for (int e = threadIdx.x; e < TX * TY; e += blockDim.x) {
    const int i = x0 + e % TX, j = y0 + e / TX;
    if (i >= L.nx || j >= L.ny) continue;
    const int k = t.c(i, j);
    if (tail == 1) {
      float off, diag; stencil_s(t, L.nx, L.ny, i, j, off, diag);
      const double r = diag <= 0.f ? 0.0 : (double)(t.rhs[k] - (off - diag * t.p[k]) / L.h2);
      part += r * r;
    } else if (tail == 2) {
      S.p64[j * L.nx + i] += (double)t.p[k];
    } else if (tail == 3) {
      // z = the cycle's p; Lz from the tile (its ring is exact after the fourth pass), in FP64
      const int kk = j * L.nx + i;
      const double z = (double)t.p[k];
      const double lz = lap_tile64(t, L, i, j, rh2);
      S.dB[kk] = lz;
      part += S.r64[kk] * z;
      part2 += S.q64[kk] * z;
      part3 += z * lz;
    }
  }
  if (tail == 3) {
    const double pa = block_sum(part, red);
    const double pb = block_sum(part2, red);
    const double pz = block_sum(part3, red);
    double ta = 0.0, tb = 0.0, tz = 0.0;
    if (scene_reduce3(S, w.tile, S.nt_up0, pa, pb, pz, red, &ta, &tb, &tz) && threadIdx.x == 0) pcg_coef(S, ta, tb, tz);
    return;
  }
  if (tail != 1) return;
  const double bpart = block_sum(part, red);
  double total = 0.0;
  if (scene_reduce(S, w.tile, S.nt_up0, bpart, red, &total) && threadIdx.x == 0) solve_decide(ctl, ss, total, true);
}

// ------------------------------------------------------------------ fused Krylov mode: the loop decision
// One CTA per scene, after the level-0 up kernel has completed: the nine sums over the scene's
// tiles (thread t adds tiles t, t + 256, ... in that order, four tiles' loads in flight at a
// time; then block_sum_t's fixed order), the cycle's coefficients and the decision. A scene
// that is disabled or no longer cycles wrote no partials and does not decide.
__global__ void __launch_bounds__(256) k_pcg_decide(const SceneDesc* __restrict__ scenes, SolveCtl* ctl) {
  const SceneDesc& S = scenes[blockIdx.x];
  pdl_trigger();
  const bool on = S.enabled;   // host-written, constant during the step
  const int nt = S.nt_up0;
  SolveState* ss = S.solve;
  pdl_wait();
  // the flag, the solve state and the partials are read together (the partial array is always
  // allocated; a scene that stopped leaves stale values, which are loaded but not used)
  const int act = *(volatile int*)&ss->active;
  PcgPrev pv{};
  DecideIn din{};
  if (threadIdx.x == 0) {
    pv = pcg_load(ss);
    din = decide_load(ctl, ss);
  }
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int k0 = threadIdx.x; k0 < nt; k0 += 4 * 256) {
    double a[4][9];
    #pragma unroll
    for (int j = 0; j < 4; j++)
      #pragma unroll
      for (int m = 0; m < 9; m++) a[j][m] = k0 + 256 * j < nt ? __ldcg(S.part + (size_t)m * nt + k0 + 256 * j) : 0.0;
    #pragma unroll
    for (int j = 0; j < 4; j++)
      if (k0 + 256 * j < nt)
        #pragma unroll
        for (int m = 0; m < 9; m++) v[m] += a[j][m];
  }
  if (!on || act == 0) return;   // the same in every thread of the CTA
  __shared__ double redt[9 * 256 + 9];
  block_sum_t<9>(v, redt);
  if (threadIdx.x == 0) {
    double alpha, beta;
    pcg_coef(ss, pv, v[0], v[1], v[2], &alpha, &beta);
    // ||r - alpha (Lz + beta q)||^2 from the dot products
    const double rq = v[4] + beta * v[5];
    const double qq = v[6] + 2.0 * beta * v[7] + beta * beta * v[8];
    const double r2 = v[3] - 2.0 * alpha * rq + alpha * alpha * qq;
    solve_decide(ctl, ss, din, r2 > 0.0 ? r2 : 0.0, true);
  }
}

// ------------------------------------------------------------------ coarse block: levels lc..coarsest in one CTA
// Shared memory holds every level >= lc with the global row pitches (pc for p,
// rhs, ay; pu for ax), so each array arrives by one TMA bulk copy; then a
// residual scratch of level lc's size.
namespace {
constexpr int CB_THREADS = 512;
constexpr int kStagedInverseMax = 128;   // coarsest unknowns whose inverse (<= 64 KB) is staged in shared memory
constexpr int CB_WARPS = CB_THREADS / 32;
constexpr int SWEEP_M = 6;              // largest coarsest level of the one-warp sweeps: rows per lane
constexpr int COARSEST_SCRATCH = 0;     // the coarsest keeps its stencils in registers
using namespace mgc;


// Cells of a level mapped linearly onto the block: thread t takes column t % w of rows
// t / w, t / w + R, ... (R = rows per round of the block), so every lane works whatever the
// level's width and warps beyond the level's cells skip at once. w > CB_THREADS: the block
// strides along each row instead.
struct LinMap {
  int i0, j0, R;   // first column and row of this thread, rows per round (0: the thread idles)
  __device__ __forceinline__ LinMap(int w, unsigned long long mw) {   // mw = fdiv_magic(w)
    if (w >= CB_THREADS) { i0 = threadIdx.x; j0 = 0; R = 1; }
    else {
      R = fdiv(CB_THREADS, mw);
      j0 = fdiv(threadIdx.x, mw);
      i0 = threadIdx.x - j0 * w;
      if (j0 >= R) R = 0;
    }
  }
  __device__ __forceinline__ int di(int w) const { return w >= CB_THREADS ? CB_THREADS : w; }   // column stride
};
// one colour pass over the cells of one colour: slot q of row j is cell i = 2q + ((j + color) & 1).
// A pass reads only cells of the other colour: up to 4 rows of a thread are computed before
// any is stored, so their shared-memory loads overlap.
__device__ __forceinline__ void pass_d(const LvS& L, int color, const LinMap& mp) {
  const int half = (L.nx + 1) >> 1;
  if (!mp.R) return;
  for (int q = mp.i0; q < half; q += mp.di(half))
    for (int jb = mp.j0; jb < L.ny; jb += 4 * mp.R) {
      float v[4];
      int kk[4];
      #pragma unroll
      for (int m = 0; m < 4; m++) {
        const int j = jb + m * mp.R, i = 2 * q + ((j + color) & 1);
        kk[m] = -1;
        if (j < L.ny && i < L.nx) {
          float off, diag; stencil_d(L, i, j, off, diag);
          const int k = j * L.pc + i;
          v[m] = diag > 0.f ? (off - L.rhs[k] * L.h2) / diag : 0.f;
          kk[m] = k;
        }
      }
      #pragma unroll
      for (int m = 0; m < 4; m++)
        if (kk[m] >= 0) L.p[kk[m]] = v[m];
    }
}
// A level visit's smoothing with every cell's stencil in registers: thread t owns colour
// slots t, t + CB_THREADS, ... (slot -> row slot / half, cell 2 (slot % half) + parity) of
// each colour, and builds their stencils once (coefficients, neighbour flags, rhs h2, the
// diagonal and its correctly rounded reciprocal) for the visit's two sweeps. The update is
// pass_d's, with the division by the diagonal as div_by_rcp: the same quotient.
// one cell's stencil in 9 registers: fl bit 0..3 = west, east, south, north neighbour present
struct RCell { float w, e, s, n, rh, diag, rcp; int kp, fl; };
// the diagonal's reciprocal comes from the block's table (L.rc, built once per kernel)
__device__ __forceinline__ RCell rcell_of(const LvS& L, int i, int j) {
  RCell c;
  c.kp = j * L.pc + i;
  c.w = L.ax[j * L.pu + i]; c.e = L.ax[j * L.pu + i + 1];
  c.s = L.ay[c.kp]; c.n = L.ay[c.kp + L.pc];
  float diag = 0.f;
  if (i > 0) diag += c.w; else diag += 2.f * c.w;
  if (i < L.nx - 1) diag += c.e; else diag += 2.f * c.e;
  if (j > 0) diag += c.s;
  if (j < L.ny - 1) diag += c.n; else diag += 2.f * c.n;
  c.diag = diag;
  c.rcp = L.rc[j * L.nx + i];
  c.rh = L.rhs[c.kp] * L.h2;
  c.fl = (i > 0 ? 1 : 0) | (i < L.nx - 1 ? 2 : 0) | (j > 0 ? 4 : 0) | (j < L.ny - 1 ? 8 : 0);
  return c;
}
// res (the down visit's residuals, or null): after the sweeps, each thread writes the residual
// of its cells (pressure.wgsl:96-101, with the stencils it holds) to res[j * pc + i]
template <int NPER>
__device__ __forceinline__ void smooth_regs(const LvS& L, int first, float* res = nullptr) {
  const int half = (L.nx + 1) >> 1;
  RCell c[2][NPER];
  bool act[2][NPER];
  #pragma unroll
  for (int col = 0; col < 2; col++)
    #pragma unroll
    for (int m = 0; m < NPER; m++) {
      const int t = threadIdx.x + m * CB_THREADS;
      const int j = fdiv(t, L.mhalf), i = 2 * (t - j * half) + ((j + col) & 1);
      act[col][m] = j < L.ny && i < L.nx;
      if (act[col][m]) c[col][m] = rcell_of(L, i, j);
    }
  #pragma unroll 1
  for (int k = 0; k < 2; k++)
    #pragma unroll
    for (int h = 0; h < 2; h++) {
      const int col = h == 0 ? first : 1 - first;
      float v[NPER];
      #pragma unroll
      for (int m = 0; m < NPER; m++) {
        if (!act[col][m]) continue;
        const RCell& q = c[col][m];
        float off = 0.f;
        if (q.fl & 1) off += q.w * L.p[q.kp - 1];
        if (q.fl & 2) off += q.e * L.p[q.kp + 1];
        if (q.fl & 4) off += q.s * L.p[q.kp - L.pc];
        if (q.fl & 8) off += q.n * L.p[q.kp + L.pc];
        v[m] = q.diag > 0.f ? div_by_rcp(off - q.rh, q.diag, q.rcp) : 0.f;
      }
      #pragma unroll
      for (int m = 0; m < NPER; m++)
        if (act[col][m]) L.p[c[col][m].kp] = v[m];
      __syncthreads();
    }
  if (!res) return;
  #pragma unroll
  for (int col = 0; col < 2; col++)
    #pragma unroll
    for (int m = 0; m < NPER; m++) {
      if (!act[col][m]) continue;
      const RCell& q = c[col][m];
      float off = 0.f;
      if (q.fl & 1) off += q.w * L.p[q.kp - 1];
      if (q.fl & 2) off += q.e * L.p[q.kp + 1];
      if (q.fl & 4) off += q.s * L.p[q.kp - L.pc];
      if (q.fl & 8) off += q.n * L.p[q.kp + L.pc];
      res[q.kp] = q.diag <= 0.f ? 0.f : L.rhs[q.kp] - div_by_rcp(off - q.diag * L.p[q.kp], L.h2, L.rh2);
    }
  __syncthreads();
}
// both sweeps of a level visit (colour `first` first in each sweep, a block barrier after
// every pass): in registers when each thread owns at most two cells of a colour. With res
// (a down visit), true when the residuals were also written there (the register path)
__device__ __forceinline__ bool smooth_visit(const LvS& L, int first, float* res = nullptr) {
  const int half = (L.nx + 1) >> 1, nslot = half * L.ny;
  if (nslot <= CB_THREADS) { smooth_regs<1>(L, first, res); return res != nullptr; }
  if (nslot <= 2 * CB_THREADS) { smooth_regs<2>(L, first, res); return res != nullptr; }
  const LinMap mh(half, L.mhalf);
  for (int k = 0; k < 2; k++) { pass_d(L, first, mh); __syncthreads(); pass_d(L, 1 - first, mh); __syncthreads(); }
  return false;
}
// The coarse block's level visits (k_mg_coarse), and what they read beside the block's shared
// memory.
struct CbCtx {
  float* smem;
  const LvO* lvo;     // level offsets in smem (shared)
  float* sres;        // residual scratch (level lc size)
  const SceneDesc* S;
  int nl, s_dir, s_inv, s_A;
};
// level l's visit on the way down: smoothing, then per coarse cell the residuals of its four
// fine cells summed in the restriction's order
__device__ __forceinline__ void cb_down(const CbCtx c, int l) {
  float* const smem = c.smem;
  const LvO* const lvo = c.lvo;
  const LvS F = lvs_at(smem, lvo[l]), Cc = lvs_at(smem, lvo[l + 1]);
  const LinMap mc(Cc.nx, Cc.mnx);
  // the residuals from the smoothing's register stencils (pitched like F in the scratch), or
  // recomputed per coarse cell on the shared-memory path of large levels
  if (smooth_visit(F, 0, c.sres)) {
    const float* r = c.sres;
    if (mc.R)
    for (int J = mc.j0; J < Cc.ny; J += mc.R)
      for (int I = mc.i0; I < Cc.nx; I += mc.di(Cc.nx)) {
        const int e = 2 * J * F.pc + 2 * I;
        Cc.rhs[J * Cc.pc + I] = 0.25f * (r[e] + r[e + 1] + r[e + F.pc] + r[e + F.pc + 1]);
        Cc.p[J * Cc.pc + I] = 0.f;
      }
    __syncthreads();
    return;
  }
  auto res = [&](int i, int j) {
    float off, diag; stencil_d(F, i, j, off, diag);
    const int e = j * F.pc + i;
    return diag <= 0.f ? 0.f : F.rhs[e] - div_by_rcp(off - diag * F.p[e], F.h2, F.rh2);
  };
  if (mc.R)
  for (int J = mc.j0; J < Cc.ny; J += mc.R)
    for (int I = mc.i0; I < Cc.nx; I += mc.di(Cc.nx)) {
      const float r = res(2 * I, 2 * J) + res(2 * I + 1, 2 * J) + res(2 * I, 2 * J + 1) + res(2 * I + 1, 2 * J + 1);
      Cc.rhs[J * Cc.pc + I] = 0.25f * r;
      Cc.p[J * Cc.pc + I] = 0.f;
    }
  __syncthreads();
}
// The 120 red-black sweeps (pressure.wgsl:132-156) in the registers of one warp, for levels up to
// 64 cells wide: lane (g, k) owns columns 2k and 2k + 1 of the M rows from M g on (M even), so one
// cell of each colour per row. A colour pass reads the other colour only: one of the west and
// east neighbours is the lane's own cell, the other a shuffle from the lane beside, the south and
// north ones are the lane's own rows', at the ends of its rows from the lanes below and above; which,
// is known at compile time from the row's parity. Bound by the latency of the 240 dependent
// passes: M + 2 shuffles and one cell's arithmetic each, where the block's pass (coarsest_update,
// kept for the sizes that do not fit) adds a store to shared memory, a barrier and loads. A missing
// neighbour's coefficient is zero and a cell without open faces has zeros throughout; with them
// and without the leading +0 of pressure.wgsl:77-85 the sums keep their values.
// Not inlined: its registers are its own, one call per coarsest solve.
// The block of a 32x48 scene (8x12 coarsest): 31.3 us by the block's passes, 22.8 with two shuffles
// per cell (a column of each lane's pairs of rows), 19.8 now.
template <int M>
__device__ __noinline__ void sweeps_warp(float* smem, const LvO& o, int W) {   // W: lanes per group, (nx + 1) / 2
  static_assert(M % 2 == 0, "a lane's first row is even");
  const LvS L = lvs_at(smem, o);
  const int lane = threadIdx.x & 31, g = lane / W, k = lane - g * W, ng = 32 / W;
  float w[2][M], e[2][M], so[2][M], no[2][M], rh[2][M], di[2][M], rc[2][M], p[2][M];
  #pragma unroll
  for (int c = 0; c < 2; c++)
    #pragma unroll
    for (int m = 0; m < M; m++) {
      const int i = 2 * k + ((m + c) & 1), j = g * M + m;
      w[c][m] = e[c][m] = so[c][m] = no[c][m] = rh[c][m] = di[c][m] = rc[c][m] = p[c][m] = 0.f;
      if (g >= ng || i >= L.nx || j >= L.ny) continue;
      const CCell q = coarsest_cell(L, j * L.nx + i);
      if (!(q.diag > 0.f)) continue;
      if (q.hw) w[c][m] = q.w;
      if (q.he) e[c][m] = q.e;
      if (q.hs) so[c][m] = q.s;
      if (q.hn) no[c][m] = q.n;
      rh[c][m] = q.rh; di[c][m] = q.diag; rc[c][m] = q.rcp;
    }
  #pragma unroll 1
  for (int it = 0; it < 120; it++)
    #pragma unroll
    for (int c = 0; c < 2; c++) {
      float (&q)[M] = p[1 - c];
      float x[M];
      #pragma unroll
      for (int m = 0; m < M; m++)
        x[m] = (m + c) & 1 ? __shfl_down_sync(0xffffffffu, q[m], 1) : __shfl_up_sync(0xffffffffu, q[m], 1);
      const float below = __shfl_sync(0xffffffffu, q[M - 1], lane - W), above = __shfl_sync(0xffffffffu, q[0], lane + W);
      #pragma unroll
      for (int m = 0; m < M; m++) {
        const bool right = (m + c) & 1;
        float off = w[c][m] * (right ? q[m] : x[m]);
        off += e[c][m] * (right ? x[m] : q[m]);
        off += so[c][m] * (m > 0 ? q[m > 0 ? m - 1 : 0] : below);
        off += no[c][m] * (m < M - 1 ? q[m < M - 1 ? m + 1 : m] : above);
        p[c][m] = div_by_rcp(off - rh[c][m], di[c][m], rc[c][m]);
      }
    }
  #pragma unroll
  for (int c = 0; c < 2; c++)
    #pragma unroll
    for (int m = 0; m < M; m++) {
      const int i = 2 * k + ((m + c) & 1), j = g * M + m;
      if (g < ng && i < L.nx && j < L.ny) L.p[j * L.pc + i] = p[c][m];
    }
}
// the coarsest level's solve (its p overwritten: the inverse's product, or sweeps from zero)
// WARP: with the one-warp sweeps (the call costs the W tail's instance, whose coarsest solve appears
// twice, 560 bytes of spill: it keeps the block's passes)
template <bool WARP>
__device__ __forceinline__ void cb_coarsest(const CbCtx c) {
  float* const smem = c.smem;
  const LvO* const lvo = c.lvo;
  float* const sres = c.sres;
  const SceneDesc& S = *c.S;
  const int nl = c.nl, s_dir = c.s_dir, s_inv = c.s_inv, s_A = c.s_A;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // ---- coarsest (pressure.wgsl:132-156): 120 red-black sweeps from zero. Row-major
    // cells 2t and 2t+1 have opposite colours for any nx (even nx: same row, adjacent;
    // odd nx: colour = index parity), so thread t owns one cell of each colour and every
    // thread works in every pass; the ceil(n/2) threads (<= 128, rounded up to warps)
    // sync on a named barrier while the other warps wait at the block barrier below.
    // Stencils, diagonals and their reciprocals stay in registers for all sweeps.
    if (s_dir) {
      // direct coarse solve (TOL/FP64 modes): p = A^-1 b with b = -rhs h2 (0 in closed cells),
      // each row's dot product as 8 strided partial sums combined pairwise (the oracle's order)
      const LvS L = lvs_at(smem, lvo[nl - 1]);
      const int n = L.nx * L.ny;
      for (int k = threadIdx.x; k < n; k += CB_THREADS) {
        const int j = fdiv(k, L.mnx), i = k - j * L.nx;
        sres[k] = L.rc[k] > 0.f ? -(L.rhs[j * L.pc + i] * L.h2) : 0.f;
      }
      __syncthreads();
      const int q = lane & 7;
      const bool staged = s_inv != 0;
      // the global copy is addressed only when the inverse is not staged
      const int ld = cinv_ld(n);
      const float* Ag = staged ? nullptr : S.cinv + (size_t)S.solve->cinv_cur * n * ld;
      const float* As = smem + s_A;
      for (int base = warp * 4; base < n; base += CB_WARPS * 4) {
        const int k = base + (lane >> 3);
        float sum = 0.f;
        if (k < n) {
          if (staged) {
            #pragma unroll 4
            for (int m = q; m < n; m += 8) sum = __fmaf_rn(As[k * ld + m], sres[m], sum);
          } else {
            #pragma unroll 4
            for (int m = q; m < n; m += 8) sum = __fmaf_rn(__ldg(Ag + (size_t)k * ld + m), sres[m], sum);
          }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (k < n && q == 0) { const int j = fdiv(k, L.mnx); L.p[j * L.pc + k - j * L.nx] = sum; }
      }
    } else {
      const LvS L = lvs_at(smem, lvo[nl - 1]);
      const int npair = (L.nx * L.ny + 1) >> 1;
      const int nthr = (npair + 31) & ~31;
      // rows a lane of the one-warp form owns
      const int W = (L.nx + 1) / 2, M = W <= 32 ? (L.ny + 32 / W - 1) / (32 / W) : SWEEP_M + 1;
      if (WARP && M <= SWEEP_M) {
        if (warp == 0) {
          if (M <= 2) sweeps_warp<2>(smem, lvo[nl - 1], W);
          else if (M <= 4) sweeps_warp<4>(smem, lvo[nl - 1], W);
          else sweeps_warp<SWEEP_M>(smem, lvo[nl - 1], W);
        }
      } else if ((int)threadIdx.x < nthr) {
        const CCell a = coarsest_cell(L, 2 * threadIdx.x), b = coarsest_cell(L, 2 * threadIdx.x + 1);
        if (a.act) L.p[a.kp] = 0.f;
        if (b.act) L.p[b.kp] = 0.f;
        // colour of cell 2t: (i + j) & 1
        const int k0 = 2 * threadIdx.x;
        const int j0 = fdiv(k0, L.mnx);
        const bool a_red = ((k0 - j0 * L.nx + j0) & 1) == 0;
        const CCell c0 = a_red ? a : b, c1 = a_red ? b : a;
        float* p = L.p;
        bar_coarsest(nthr);
        #pragma unroll 1
        for (int it = 0; it < 120; it++) {
          coarsest_update(p, L.pc, c0);
          bar_coarsest(nthr);
          coarsest_update(p, L.pc, c1);
          bar_coarsest(nthr);
        }
      }
    }
    __syncthreads();
}
// level l's visit on the way up: prolongation of level l + 1's p, then smoothing
__device__ __forceinline__ void cb_up(const CbCtx c, int l) {
  float* const smem = c.smem;
  const LvO* const lvo = c.lvo;
    const LvS F = lvs_at(smem, lvo[l]), Cc = lvs_at(smem, lvo[l + 1]);
    const LinMap mp(F.nx, F.mnx);
    if (mp.R)
    for (int j = mp.j0; j < F.ny; j += mp.R)
      for (int i = mp.i0; i < F.nx; i += mp.di(F.nx)) {
        const int I = i / 2, J = j / 2;
        const int I2 = min(max(I + ((i & 1) == 1 ? 1 : -1), 0), Cc.nx - 1);
        const int J2 = min(max(J + ((j & 1) == 1 ? 1 : -1), 0), Cc.ny - 1);
        const float c = 0.5625f * Cc.p[J * Cc.pc + I] + 0.1875f * (Cc.p[J * Cc.pc + I2] + Cc.p[J2 * Cc.pc + I]) +
                        0.0625f * Cc.p[J2 * Cc.pc + I2];
        F.p[j * F.pc + i] += F.rc[j * F.nx + i] > 0.f ? c : 0.f;
      }
    __syncthreads();
    smooth_visit(F, 1);
}
}  // namespace

// smem_floats: the launch's dynamic shared memory in floats; past the levels and the residual
// scratch, the coarsest inverse of the direct solve is staged there when it fits
// WT: compiled with the W tail (an engine whose scenes have one); without it the V-cycle's code alone
// L0: compiled with the level-0 ends of the cycle (an engine where some scene's block covers level 0)
template <bool WT, bool L0>
__global__ void __launch_bounds__(CB_THREADS) k_mg_coarse(const SceneDesc* __restrict__ scenes, int nscenes, SolveCtl* ctl, int tail,
                                                         int count_iter, int smem_floats) {
  extern __shared__ __align__(128) float smem[];
  __shared__ double red[32];
  __shared__ LvO lvo[MAX_LEVELS];
  __shared__ __align__(8) uint64_t bar;    // the coefficients (+ inverse)
  __shared__ int s_idle;                          // as in k_mg_down
  __shared__ int s_inv, s_res, s_A, s_dir, s_gpc;   // offsets: residual scratch, inverse
  __shared__ float* s_gp;                         // level lc's p in global memory
  const SceneDesc& S = scenes[blockIdx.x];
  pdl_trigger();
  const int lc = S.lc, nl = S.nlev;
  if (threadIdx.x == 0) {
    int q = 0;
    for (int l = lc; l < nl; l++) {
      const LevelDesc& G = S.lev[l];
      LvS v;
      v.nx = G.nx; v.h2 = G.h2; lvs_derive(v);
      LvO o;
      o.nx = G.nx; o.ny = G.ny; o.pc = G.pc; o.pu = G.pu; o.h2 = G.h2; o.rh2 = v.rh2; o.mnx = v.mnx; o.mhalf = v.mhalf;
      o.po = q; q += G.ny * G.pc;
      o.ro = q; q += G.ny * G.pc;
      o.ao = q; q += G.ny * G.pu;
      o.yo = q; q += (G.ny + 1) * G.pc;
      lvo[l] = o;
    }
    s_res = q;
    const int nres = S.lev[lc].ny * S.lev[lc].pc;   // the largest level's pitched size
    q += round_up(nres > COARSEST_SCRATCH ? nres : COARSEST_SCRATCH, 32);   // residual scratch
    for (int l = lc; l < nl; l++) { lvo[l].to = q; q += S.lev[l].nx * S.lev[l].ny; }
    q = round_up(q, 32);
    s_A = q;
    s_gp = S.lev[lc].p; s_gpc = S.lev[lc].pc;
    s_idle = scene_idle(S.solve);
    mbar_init(&bar, 1);
  }
  __syncthreads();
  // ---- stage the arrays. The coefficients are built before the pressure loop and no loop
  // kernel writes them; the direct solve's inverse (the half cinv_cur of S.cinv) is factored
  // before the loop or, pipelined, during the previous step (this step's side branch writes
  // the other half). Both arrive by TMA bulk copies (sizes multiples of 16 bytes; the
  // inverse when it fits, n even) before the wait on the previous kernel, and the reciprocal
  // of each cell's diagonal (pressure.wgsl:77-86; 0 marks a closed cell) is tabled then too,
  // beside the previous kernel. After the wait only level lc's rhs (and p when lc = 0) is
  // read, with plain loads from L2.
  const volatile int* act = &S.solve->active;
  const bool on = S.enabled && !s_idle;   // enabled: host-written, constant during the step
  if (threadIdx.x == 0) {
    s_inv = 0;
    s_dir = 0;
    if (on) {
      uint32_t bytes = 0;
      for (int l = lc; l < nl; l++) bytes += (S.lev[l].ny * S.lev[l].pu + (S.lev[l].ny + 1) * S.lev[l].pc) * 4;
      const int n = S.lev[nl - 1].nx * S.lev[nl - 1].ny;
      s_dir = ctl->coarse_direct && S.solve->direct_ok;   // both fixed for the loop
      const int ld = cinv_ld(n);
      const bool inv = s_dir && (n % 2) == 0 && n <= kStagedInverseMax && s_A + n * ld <= smem_floats;
      if (inv) bytes += (uint32_t)(n * ld * 4);
      mbar_arrive_expect_tx(&bar, bytes);
      for (int l = lc; l < nl; l++) {
        const LevelDesc& G = S.lev[l];
        bulk_g2s(smem + lvo[l].ao, G.ax, G.ny * G.pu * 4, &bar);
        bulk_g2s(smem + lvo[l].yo, G.ay, (G.ny + 1) * G.pc * 4, &bar);
      }
      if (inv) {
        bulk_g2s(smem + s_A, S.cinv + (size_t)S.solve->cinv_cur * n * ld, (uint32_t)(n * ld * 4), &bar);
        s_inv = 1;
      }
    }
  }
  const LvS V0 = lvs_at(smem, lvo[lc]);
  const float* grhs = S.lev[lc].rhs;
  bool okc = true;
  if (on) {
    okc = mbar_wait(&bar, 0);
    if (okc)
      for (int l = lc; l < nl; l++) {
        const LvS L = lvs_at(smem, lvo[l]);
        float* rc = smem + lvo[l].to;
        for (int e = threadIdx.x; e < L.nx * L.ny; e += CB_THREADS) {
          const int j = fdiv(e, L.mnx), i = e - j * L.nx;
          const float d = diag_d(L, i, j);
          rc[e] = d > 0.f ? __frcp_rn(d) : 0.f;
        }
      }
    // level lc's p is zero after the restriction into it (pressure.wgsl:112)
    if (lc > 0)
      for (int e = threadIdx.x; e < V0.ny * V0.pc; e += CB_THREADS) V0.p[e] = 0.f;
  }
  pdl_wait();
  if (count_iter && blockIdx.x == 0 && threadIdx.x == 0) loop_count(ctl);
  if (!on) return;
  if (__syncthreads_or(!okc)) {
    // the copies did not land in time: record it and leave once they have (bounded)
    if (threadIdx.x == 0) atomicExch(&ctl->err, 1);
    mbar_wait(&bar, 0);
    return;
  }
  // the scene's flag and level lc's rhs are read together (two L2 round trips overlapped): the
  // loads land in shared memory whether or not the scene still cycles, then every thread leaves
  // together if it does not
  const int still = *act;
  float* sres = smem + s_res;   // residual scratch (level lc size)
  for (int e = threadIdx.x; e < V0.ny * V0.pc; e += CB_THREADS) V0.rhs[e] = __ldcg(grhs + e);
  if (L0 && lc == 0)   // warm start
    for (int e = threadIdx.x; e < V0.ny * V0.pc; e += CB_THREADS) V0.p[e] = __ldcg(s_gp + e);
  if (still == 0) return;
  __syncthreads();
  const CbCtx cbx{smem, lvo, sres, &S, nl, s_dir, s_inv, s_A};
  // The cycle over levels lc..nl-1: the V(2,2) cycle of js/fluid.js:294-312, straight down, the
  // coarsest, straight up. With the W tail (S.lw = nl - 3) level nl - 3 visits level nl - 2
  // twice: after the first visit has come back up through level nl - 2, that level is smoothed
  // from its p and restricted again (its rhs stays) and the coarsest solved again. Straight-line
  // code: the visits keep their registers to themselves.
  for (int l = lc; l < nl - 1; l++) cb_down(cbx, l);
  cb_coarsest<!WT>(cbx);
  if (WT && S.lw == nl - 3 && nl - 3 >= lc) {
    cb_up(cbx, nl - 2);
    cb_down(cbx, nl - 2);
    cb_coarsest<!WT>(cbx);
  }
  for (int l = nl - 2; l >= lc; l--) cb_up(cbx, l);
  // ---- write level lc back; when the block covers level 0, finish the cycle here
  float* const gp = s_gp;
  const int gpc = s_gpc, gnx = V0.nx;
  if (!L0 || lc > 0) {
    // the shared copy of level lc's p has the global pitch: one bulk copy (the last visit ended
    // with a block barrier); the next kernel reads it after this grid has completed
    if (threadIdx.x == 0) {
      proxy_fence_shared();
      bulk_s2g(gp, V0.p, (uint32_t)(V0.ny * gpc * 4));
      bulk_wait_read();
    }
    return;
  }
  double part = 0.0, part2 = 0.0, part3 = 0.0;
  const LinMap mw(V0.nx, V0.mnx);
  if (mw.R)
  for (int j = mw.j0; j < V0.ny; j += mw.R)
    for (int i = mw.i0; i < V0.nx; i += mw.di(V0.nx)) {
      const int e = j * V0.pc + i;
      gp[j * gpc + i] = V0.p[e];
      if (lc == 0 && tail == 1) {
        float off, diag; stencil_d(V0, i, j, off, diag);
        const double r = diag <= 0.f ? 0.0 : (double)(V0.rhs[e] - (off - diag * V0.p[e]) / V0.h2);
        part += r * r;
      } else if (lc == 0 && tail == 2) {
        S.p64[j * gnx + i] += (double)V0.p[e];
      } else if (lc == 0 && tail == 3) {
        const double z = (double)V0.p[e];
        const double lz = lap_block64(V0, i, j);
        S.dB[j * gnx + i] = lz;
        part += S.r64[j * gnx + i] * z;
        part2 += S.q64[j * gnx + i] * z;
        part3 += z * lz;
      }
    }
  if (lc == 0 && tail == 1) {
    const double t = block_sum(part, red);
    if (threadIdx.x == 0) solve_decide(ctl, S.solve, t, true);
  } else if (lc == 0 && tail == 3) {
    const double ta = block_sum(part, red);
    const double tb = block_sum(part2, red);
    const double tz = block_sum(part3, red);
    if (threadIdx.x == 0) pcg_coef(S, ta, tb, tz);
  }
}

// ------------------------------------------------------------------ direct coarse solve: the coarsest inverse
// The coarsest operator A (A_kk = the stencil's diagonal, A_km = -face coefficient;
// a closed cell gets the row dmax e_k) is symmetric with half-bandwidth nx in
// row-major cell order. Once per step: banded Cholesky A = L L^T (right-looking,
// one warp: per column jc, L_jcjc = sqrt(a_jcjc), L_ijc = a_ijc / L_jcjc, then
// a_ik = fma(-L_ijc, L_kjc, a_ik) for jc < k <= i <= jc + nx), then column c of
// A^-1 by forward and back substitution on thread c (y_i = (e_ic - sum L_ik y_k) *
// (1/L_ii) with k ascending, then x_i = (y_i - sum L_ki x_k) * (1/L_ii), k ascending).
// A pivot a_jcjc <= 1e-6 dmax (a sealed gas pocket: singular) or a level wider than
// CF_MAXBW cells leaves direct_ok = 0, and the coarse block keeps the 120 sweeps.
namespace {
constexpr int CF_THREADS = 256;   // the coarsest level has at most 256 cells
constexpr int CF_MAXBW = 32;
constexpr size_t CF_SMEM_BUDGET = 200 * 1024;
}

// Columns of the inverse solved per pass: all n when the working columns fit the
// shared-memory budget beside the band, else 128 per pass.
constexpr int CF_ROW = 2 * CF_MAXBW + 5;   // floats per row beside its columns: the widest band, the column, 1 / L_ii
__host__ __device__ inline int coarse_factor_cols(int n) {
  return (size_t)n * (n + CF_ROW) * sizeof(float) <= CF_SMEM_BUDGET ? n : 128;
}
size_t coarse_factor_smem(int n) { return (size_t)n * (coarse_factor_cols(n) + CF_ROW) * sizeof(float); }

// The inverse of the coarsest operator of each scene: the banded matrix is factored L L^T by one
// warp whose lanes hold the rows of the trailing band in registers (a row enters BWM columns before
// its own; the new column's l_kj by shuffle), then each thread solves L L^T x = e_c for its column
// c: forward with the next BWM rows' sums in registers, each y_i subtracted from all of them at
// once, backward with the last BWM x in registers; the forward result is kept in shared memory
// (Y[i * C + t]). Padded with zeros to BWM, rows of the band and columns of L are plain 16-byte
// loads; a zero coefficient changes no sum. Bound by latency: a warp's chain of square root, quotient
// and shuffle per column, then of one fused multiply-add per band entry and row. With the band
// packed and every load behind its own bounds test an inverse of 8x12 took 58 us, of 12x17 216, of
// 16x16 500; now 33, 111 and 113.
// pipelined = 0: the inverse of this step's operator into the half the cycles use (direct_ok);
// pipelined = 1: into the other half for the next step (direct_ok_next), while this step's
// cycles use the current half.
template <int BWM>
__global__ void __launch_bounds__(CF_THREADS) k_coarse_factor(const SceneDesc* __restrict__ scenes, int pipelined) {
  extern __shared__ float cf_smem[];
  __shared__ float s_dmax;
  __shared__ int s_ok;
  const SceneDesc& S = scenes[blockIdx.x];
  if (!S.enabled) return;
  const LevelDesc L = S.lev[S.nlev - 1];
  constexpr int WS = BWM + 4;
  const int n = L.nx * L.ny, bw = L.nx;
  int* ok_flag = pipelined ? &S.solve->direct_ok_next : &S.solve->direct_ok;
  const int ld = cinv_ld(n);
  float* cinv = S.cinv + (size_t)(pipelined ? 1 - S.solve->cinv_cur : S.solve->cinv_cur) * n * ld;
  if (n > CF_THREADS || bw > BWM) {
    if (threadIdx.x == 0) *ok_flag = 0;
    return;
  }
  // L below A in place: band[i * WS + m] = A[i][i - BWM + m], the diagonal at m = BWM, zeros left of the band
  float* band = cf_smem;                 // n * WS
  float* col = band + n * WS;            // n * BWM: col[i * BWM + m] = L[i + 1 + m][i]
  float* rinv = col + n * BWM;           // n
  float* Y = rinv + n;                   // n * C
  const int C = coarse_factor_cols(n);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < n * WS; e += CF_THREADS) band[e] = 0.f;
  __syncthreads();
  // the diagonal is kept in rinv[] until dmax is known
  for (int k = tid; k < n; k += CF_THREADS) {
    const int i = k % L.nx, j = k / L.nx;
    const float w = L.ax[j * L.pu + i], e = L.ax[j * L.pu + i + 1];
    const float so = L.ay[j * L.pc + i], no = L.ay[(j + 1) * L.pc + i];
    float diag = 0.f;
    if (i > 0) diag += w; else diag += 2.f * w;
    if (i < L.nx - 1) diag += e; else diag += 2.f * e;
    if (j > 0) diag += so;
    if (j < L.ny - 1) diag += no; else diag += 2.f * no;
    rinv[k] = diag;
    if (diag > 0.f) {
      float* r = band + k * WS + BWM;
      r[0] = diag;
      if (i > 0) r[-1] = -w;
      if (j > 0) r[-bw] = -so;
    }
  }
  __syncthreads();
  if (warp == 0) {
    float m = 0.f;
    for (int k = lane; k < n; k += 32) m = fmaxf(m, rinv[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) { s_dmax = m; s_ok = m > 0.f ? 1 : 0; }
  }
  __syncthreads();
  const float dmax = s_dmax, thr = 1e-6f * dmax;
  for (int k = tid; k < n; k += CF_THREADS)
    if (!(rinv[k] > 0.f)) band[k * WS + BWM] = dmax;
  __syncthreads();
  if (warp == 0 && s_ok) {
    // row i lives in lane i % 32 from column i - BWM on: a[m] = A[i][jc + m]; in: the row that enters next
    float a[WS], in[WS];
    auto row = [&](int i, float (&v)[WS]) {
      const float4* r = reinterpret_cast<const float4*>(band + min(i, n - 1) * WS);
#pragma unroll
      for (int m = 0; m < WS / 4; m++) { const float4 q = r[m]; v[4 * m] = q.x; v[4 * m + 1] = q.y; v[4 * m + 2] = q.z; v[4 * m + 3] = q.w; }
    };
    row(lane, in);
#pragma unroll
    for (int m = 0; m <= BWM; m++) a[m] = in[m];
    // row r < BWM starts at column 0: its first BWM - r entries lie left of the matrix
    for (int r = lane; r < BWM; r++) {
#pragma unroll
      for (int m = 0; m < BWM; m++) a[m] = a[m + 1];
    }
    row(BWM, in);
    for (int jc = 0; jc < n; jc++) {
      const float piv = __shfl_sync(0xffffffffu, a[0], jc & 31);
      if (!(piv > thr)) {   // every lane has the same pivot
        if (lane == 0) s_ok = 0;
        break;
      }
      const bool enters = lane == ((jc + BWM) & 31);
#pragma unroll
      for (int m = 0; m <= BWM; m++) a[m] = enters ? in[m] : a[m];
      row(jc + 1 + BWM, in);
      const float ljj = sqrtf(piv);
      const int d = 1 + ((lane - jc - 1) & 31), i = jc + d;
      const bool mine = d <= bw && i < n;
      const float q = a[0] / ljj, lij = mine ? q : 0.f;
      if (lane == 0) band[jc * WS + BWM] = ljj;
      if (mine) band[i * WS + BWM - d] = lij;
      // A[i][k] -= l_ij l_kj for k = jc + 1 + m <= i (the entries past i are never read), l_kj from row k's
      // lane; zeros in the lanes of no such row
#pragma unroll
      for (int m = 0; m < BWM; m++) a[m] = __fmaf_rn(-lij, __shfl_sync(0xffffffffu, lij, (jc + 1 + m) & 31), a[m + 1]);
    }
  }
  __syncthreads();
  if (!s_ok) {
    if (tid == 0) *ok_flag = 0;
    return;
  }
  for (int k = tid; k < n; k += CF_THREADS) rinv[k] = 1.0f / band[k * WS + BWM];
  for (int e = tid; e < n * BWM; e += CF_THREADS) {
    const int i = e / BWM, m = e % BWM;
    col[e] = i + 1 + m < n ? band[(i + 1 + m) * WS + BWM - 1 - m] : 0.f;
  }
  __syncthreads();
  for (int c0 = 0; c0 < n; c0 += C) {
    const int c = c0 + tid;
    if (tid < C && c < n) {
      float* y = Y + tid;   // y[i * C]
      // rows above the warp's first column hold zeros
      const int first = c0 + (tid & ~31);
      float l[BWM], v[BWM + 1];
      auto column = [&](int i) {
        const float4* r = reinterpret_cast<const float4*>(col + i * BWM);
#pragma unroll
        for (int m = 0; m < BWM / 4; m++) { const float4 q = r[m]; l[4 * m] = q.x; l[4 * m + 1] = q.y; l[4 * m + 2] = q.z; l[4 * m + 3] = q.w; }
      };
      // forward: y_i = v_i / L[i][i], then v_k -= L[k][i] y_i for k = i+1 .. i+bw; v[m] is row i+m's sum
#pragma unroll
      for (int m = 0; m <= BWM; m++) v[m] = first + m == c ? 1.f : 0.f;
      for (int i = first; i < n; i++) {
        column(i);
        const float yi = v[0] * rinv[i];
        y[i * C] = yi;
#pragma unroll
        for (int m = 0; m < BWM; m++) v[m] = __fmaf_rn(-l[m], yi, v[m + 1]);
        v[BWM] = i + 1 + BWM == c ? 1.f : 0.f;
      }
      // backward: x_i = (y_i - sum_{k = i+1}^{min(n-1, i+bw)} L[k][i] x_k) / L[i][i], k ascending;
      // v[m] = x_{i+1+m}
#pragma unroll
      for (int m = 0; m < BWM; m++) v[m] = 0.f;
      for (int i = n - 1; i >= 0; i--) {
        column(i);
        float x = i >= first ? y[i * C] : 0.f;
#pragma unroll
        for (int m = 0; m < BWM; m++) x = __fmaf_rn(-l[m], v[m], x);
        x *= rinv[i];
        cinv[(size_t)i * ld + c] = x;
#pragma unroll
        for (int m = BWM - 1; m > 0; m--) v[m] = v[m - 1];
        v[0] = x;
      }
    }
    __syncthreads();
  }
  if (tid == 0) *ok_flag = 1;
}

// Pipelined coarse solve, after the step's pressure loop and the factorisation have both
// finished: the next step's cycles use the inverse just factored.
__global__ void k_cinv_swap(const SceneDesc* __restrict__ scenes, int nscenes) {
  for (int s = threadIdx.x; s < nscenes; s += blockDim.x) {
    const SceneDesc& S = scenes[s];
    if (!S.enabled) continue;
    SolveState* ss = S.solve;
    ss->cinv_cur ^= 1;
    ss->direct_ok = ss->direct_ok_next;
    ss->direct_ok_next = 0;
  }
}

// shared bytes of the coarse block for one scene (the layout built by k_mg_coarse)
size_t coarse_smem_bytes(const int* lnx, const int* lny, int lc, int nlev) {
  size_t f = 0;
  for (int l = lc; l < nlev; l++) {
    const size_t pc = (size_t)round_up(lnx[l], 32), pu = (size_t)round_up(lnx[l] + 1, 32);
    f += 2 * lny[l] * pc + lny[l] * pu + (lny[l] + 1) * pc;
  }
  f += (size_t)round_up(std::max(round_up(lnx[lc], 32) * lny[lc], COARSEST_SCRATCH), 32);
  size_t cells = 0;   // the 1/diag table of every level
  for (int l = lc; l < nlev; l++) cells += (size_t)lnx[l] * lny[l];
  f += (size_t)round_up((int)cells, 32);
  // room for the coarsest inverse of the direct solve when it fits
  const size_t n = (size_t)lnx[nlev - 1] * lny[nlev - 1];
  const size_t ld = (size_t)cinv_ld((int)n);
  if (n % 2 == 0 && n <= (size_t)kStagedInverseMax && (f + n * ld) * 4 <= kCoarseSmemMax) f += n * ld;
  return f * 4;
}

using UpKernel = void (*)(const SceneDesc*, int, const Work*, int, SolveCtl*, f2);
constexpr f2 kNegZero2 = 0x8000000080000000ull;
template <bool ONE>
static UpKernel up_kernel(int tail) {
  switch (tail) {
    case 1: return k_mg_up<MGF_TX, MGF_TY, 1, ONE>;
    case 2: return k_mg_up<MGF_TX, MGF_TY, 2, ONE>;
    case 3: return k_mg_up<MGF_TX, MGF_TY, 3, ONE>;
    case 4: return k_mg_up<MGF_TX, MGF_TY, 4, ONE>;
    default: return k_mg_up<MGF_TX, MGF_TY, 0, ONE>;
  }
}
// whether `ntiles` CTAs fit in one wave at two per SM (this process's device)
static bool one_wave_at_two(int ntiles) {
  static const int sms = [] {
    int d = 0, n = 0;
    if (cudaGetDevice(&d) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess)
      n = 0;
    return n;
  }();
  return ntiles <= 2 * sms;
}
void launch_mg_down(const SceneDesc* scenes, int nscenes, const Work* work, int ntiles, int level, SolveCtl* ctl,
                    int count_iter, int pcg, bool pdl, cudaStream_t st) {
  if (ntiles <= 0) return;
  const auto k = nscenes == 1
                     ? (pcg ? (one_wave_at_two(ntiles) ? k_mg_down<MGF_TX, MGF_TY, true, true, 2>
                                                       : k_mg_down<MGF_TX, MGF_TY, true, true>)
                            : k_mg_down<MGF_TX, MGF_TY, false, true>)
                     : (pcg ? k_mg_down<MGF_TX, MGF_TY, true, false> : k_mg_down<MGF_TX, MGF_TY, false, false>);
  launch_pdl(pdl && pdl_enabled(), k, dim3(ntiles), dim3(256), 0, st, scenes, nscenes, work, level, ctl, count_iter, kNegZero2);
}
void launch_mg_up(const SceneDesc* scenes, int nscenes, const Work* work, int ntiles, int level, int tail, SolveCtl* ctl,
                  cudaStream_t st) {
  if (ntiles <= 0) return;
  const UpKernel k = nscenes != 1 ? up_kernel<false>(tail)
                     : tail == 4 && one_wave_at_two(ntiles) ? k_mg_up<MGF_TX, MGF_TY, 4, true, 2>
                                                            : up_kernel<true>(tail);
  launch_pdl(pdl_enabled(), k, dim3(ntiles), dim3(256), 0, st, scenes, nscenes, work, level, ctl, kNegZero2);
}
void launch_pcg_decide(const SceneDesc* scenes, int nscenes, SolveCtl* ctl, cudaStream_t st) {
  if (nscenes > 0) launch_pdl(pdl_enabled(), k_pcg_decide, dim3(nscenes), dim3(256), 0, st, scenes, ctl);
}
void launch_mg_coarse(const SceneDesc* scenes, int nscenes, SolveCtl* ctl, int tail, int count_iter, size_t smem,
                      int wtail, int level0, bool pdl, cudaStream_t st) {
  if (nscenes > 0)
    launch_pdl(pdl && pdl_enabled(),
               wtail ? (level0 ? k_mg_coarse<true, true> : k_mg_coarse<true, false>)
                     : (level0 ? k_mg_coarse<false, true> : k_mg_coarse<false, false>),
               dim3(nscenes), dim3(CB_THREADS), smem, st, scenes, nscenes, ctl, tail, count_iter, (int)(smem / 4));
}
// bw: the widest coarsest level of the batch (the register window's bound)
void launch_coarse_factor(const SceneDesc* scenes, int nscenes, size_t smem, int bw, int pipelined, cudaStream_t st) {
  if (nscenes <= 0) return;
  if (bw <= 8) k_coarse_factor<8><<<nscenes, CF_THREADS, smem, st>>>(scenes, pipelined);
  else if (bw <= 16) k_coarse_factor<16><<<nscenes, CF_THREADS, smem, st>>>(scenes, pipelined);
  else k_coarse_factor<32><<<nscenes, CF_THREADS, smem, st>>>(scenes, pipelined);
}
void launch_cinv_swap(const SceneDesc* scenes, int nscenes, cudaStream_t st) {
  if (nscenes > 0) k_cinv_swap<<<1, 128, 0, st>>>(scenes, nscenes);
}
// The attribute belongs to the kernel, not to an engine: it is set to the largest size any
// coarsest level can ask for, so engines of different sizes never lower it under each other.
cudaError_t prepare_coarse_factor(size_t smem) {
  const int cap = (int)std::max(smem, CF_SMEM_BUDGET);   // every level that fits: the columns' budget bounds it
  cudaError_t e = cudaFuncSetAttribute(k_coarse_factor<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_coarse_factor<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_coarse_factor<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  return e;
}
cudaError_t prepare_mg_coarse(size_t smem) {
  // the kernel's attribute, shared by every engine: the largest size any schedule can ask for
  const int bytes = (int)std::max(smem, kCoarseSmemMax);
  cudaError_t e = cudaFuncSetAttribute(k_mg_coarse<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mg_coarse<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mg_coarse<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mg_coarse<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e;
}

}  // namespace cfg
