// Volume rendering of a simulation's state, headless: restates the renderer's compute passes
// (src/engine/shaders/lighting.wgsl smoothSmoke 69-99, buildOccupancy 149-244, incidentLight
// 257-310, lightSlot 312-347) and the camera march (volume-march.wgsl fireProRay 18-24,
// fireProHit 28-35, fireProStep 77-79, fireProJitter 94-102, fireProShade 106-138,
// fireProDirect 141-146, fireProMarch 178-268; scene-volume.wgsl 39-44 and 160-167 with no
// scene depth and half resolution off), the optical model (fire-emission.wgsl) and the
// reconstruction filters (volume-reconstruction.wgsl).
//
// Where the reference reads a pool slot's apron (a copy of the +1 neighbours), these kernels
// read the neighbour's slot; a neighbour without a slot reads what the apron would hold: the
// smoothed density computed on the spot for the render field, the incident light computed on
// the spot for the lighting pool. The render marches one box per cluster of tiles that holds
// content or sources (FluidSimulation.ts:916-957, TileDirectory.ts:189-245): a sample reads the
// pages of the box it lies in only, clamped to that box, and a ray crosses the boxes in order
// (volume-march.wgsl fireProSpan, fireProNext, fireProEnter).
#include "fp_device.cuh"
#include "fp_render.h"

#include <type_traits>

namespace {

constexpr int RTHREADS = 128;
// Resident CTAs an SM the march is compiled for (168 registers): four (128, spills) and five lost
// 7 % and 20 % on the slice pass, two 15 %.
constexpr int MARCH_CTAS = 3;

// A thread's current box, the bricks its samples read, and how it finds a brick's slot: through the
// boxes' tables, or (no tables, FpRender::pages null) through the tile hash. What follows is compiled for
// each, so that neither's kernels hold the other's code: one cursor that asks at each lookup took the
// hash form 10.6 ms for 231,401 rays of 700 bricks, 7.5 for 129,600 of a 1.8k-brick jet and 24.7 for
// 518,400 of 3.7k bricks (now 6.5, 4.5 and 22.8), the tables 0.95, 0.95 and 4.2 ms (0.87, 0.89, 3.8).
// Remembering the last two lookups loses: lanes that hit wait for those that miss (24.7 -> 25.9 ms).
struct TableCursor {
  int lo[3], hi[3];  // in bricks, inclusive
  int first;         // its first entry in FpRender::pages
};
struct HashCursor {
  int lo[3], hi[3];
};
template <class Cursor>
FP_DEV Cursor noBox() {
  Cursor c;
  for (int a = 0; a < 3; a++) {
    c.lo[a] = 0;
    c.hi[a] = -1;
  }
  if constexpr (std::is_same_v<Cursor, TableCursor>) c.first = 0;
  return c;
}
// Box k becomes the current one.
template <class Cursor>
FP_DEV void useBox(const FpRender& R, Cursor& c, int k) {
  for (int a = 0; a < 3; a++) {
    c.lo[a] = R.boxes[FP_BOX_INTS * k + a];
    c.hi[a] = R.boxes[FP_BOX_INTS * k + 3 + a];
  }
  if constexpr (std::is_same_v<Cursor, TableCursor>) c.first = R.boxes[FP_BOX_INTS * k + 6];
}
template <class Cursor>
FP_DEV bool inBox(const Cursor& c, int bx, int by, int bz) {
  return bx >= c.lo[0] && bx <= c.hi[0] && by >= c.lo[1] && by <= c.hi[1] && bz >= c.lo[2] && bz <= c.hi[2];
}
// The slot of world brick b, or -1, through the tile hash.
FP_DEV int hashedSlot(const SimParams& P, int bx, int by, int bz) {
  int t = hashFind(P, bx >> 2, by >> 2, bz >> 2);
  if (t < 0) return -1;
  return checkSlot(P, FP_SITE_ENTRY, entryPage(P.entries[t * 64 + (((bz & 3) * 4 + (by & 3)) * 4 + (bx & 3))]));
}
// The entry of brick b of the current box in its table.
FP_DEV int pageIndex(const TableCursor& c, int bx, int by, int bz) {
  return c.first + ((bz - c.lo[2]) * (c.hi[1] - c.lo[1] + 1) + (by - c.lo[1])) * (c.hi[0] - c.lo[0] + 1) + (bx - c.lo[0]);
}
// fireProPage: the slot of world brick b inside the current box, or less than 0 (FpRender::pages).
FP_DEV int slotAt(const SimParams& P, const FpRender& R, TableCursor& c, int bx, int by, int bz) {
  if (!inBox(c, bx, by, bz)) return -1;
  return __ldg(&R.pages[pageIndex(c, bx, by, bz)]);
}
FP_DEV int slotAt(const SimParams& P, const FpRender&, HashCursor& c, int bx, int by, int bz) {
  return inBox(c, bx, by, bz) ? hashedSlot(P, bx, by, bz) : -1;
}
// Of a low-face cell (lx,ly,lz) of a brick of `side` cells a side, its place in the brick's three
// apron planes.
FP_DEV int apronIndex(int side, int lx, int ly, int lz) {
  if (lx == 0) return lz * side + ly;
  if (ly == 0) return (side + lz) * side + lx;
  return (2 * side + ly) * side + lx;
}
// The cell at place i of a brick's apron planes; false for a place that stands for none (a cell on
// two faces has one place) and for cells that no sample based in a slotted brick reads: `before`
// has bit k set when the brick k's set bits (x, y, z) before this one on those axes has a slot.
FP_DEV bool apronCell(int side, int i, unsigned before, int& lx, int& ly, int& lz) {
  const int face = i / (side * side), a = i % side, b = (i / side) % side;
  lx = face == 0 ? 0 : a;
  ly = face == 1 ? 0 : (face == 0 ? a : b);
  lz = face == 2 ? 0 : b;
  if ((face >= 1 && lx == 0) || (face == 2 && ly == 0)) return false;
  const unsigned on = (lx == 0 ? 1u : 0u) | (ly == 0 ? 2u : 0u) | (lz == 0 ? 4u : 0u);
  for (unsigned k = 1; k < 8; k++)
    if ((k & ~on) == 0u && ((before >> k) & 1u)) return true;
  return false;
}
template <class Cursor>
FP_DEV unsigned slottedBefore(const SimParams& P, const FpRender& R, Cursor& c, int bx, int by, int bz) {
  unsigned before = 0;
  for (int k = 1; k < 8; k++)
    if (slotAt(P, R, c, bx - (k & 1), by - ((k >> 1) & 1), bz - (k >> 2)) >= 0) before |= 1u << k;
  return before;
}
// The slots of the bricks that the cells from (x,y,z) to n further on each axis lie in: s[k] for
// the low (bit clear) or high (bit set) brick on x, y, z (bits 0, 1, 2). n is less than a brick,
// `sh` the log2 of a brick's cells on the lattice asked about. False unless every one lies in the
// current box and has a slot. The common case of a sample: its taps then need no lookup each.
FP_DEV bool slots8(const FpRender&, const HashCursor&, int, int, int, int, int, int*) { return false; }
FP_DEV bool slots8(const FpRender& R, const TableCursor& c, int sh, int x, int y, int z, int n, int* s) {
  const int bx = x >> sh, by = y >> sh, bz = z >> sh, ex = (x + n) >> sh, ey = (y + n) >> sh, ez = (z + n) >> sh;
  if (bx < c.lo[0] || by < c.lo[1] || bz < c.lo[2] || ex > c.hi[0] || ey > c.hi[1] || ez > c.hi[2])
    return false;
  const int nx = c.hi[0] - c.lo[0] + 1, nxy = nx * (c.hi[1] - c.lo[1] + 1);
  const int* p = R.pages + pageIndex(c, bx, by, bz);
  const int dx = ex - bx, dy = ey != by ? nx : 0, dz = ez != bz ? nxy : 0;
  int all = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    s[k] = __ldg(p + ((k & 1) ? dx : 0) + ((k & 2) ? dy : 0) + ((k & 4) ? dz : 0));
    all |= s[k];
  }
  return all >= 0;
}

FP_DEV float glowOf(float life) { return fminf(fmaxf(life * 5.f, 0.f), 1.f); }  // fireProGlow

// The simulation's smoke at a world cell: zero outside the box or without a slot.
template <class Cursor>
FP_DEV float rawSmoke(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z) {
  int s = slotAt(P, R, c, x >> P.shift, y >> P.shift, z >> P.shift);
  if (s < 0) return 0.f;
  return ldHalf(P.fld, (size_t)s * 4 * P.N + localCell(P, x, y, z), P.scalarHalf != 0);
}
// fireProField of the smoke at `q` in cells: clamped to the box, trilinear.
template <class Cursor>
FP_DEV float smokeSample(const SimParams& P, const FpRender& R, Cursor& c, float qx, float qy, float qz) {
  float B = (float)P.B;
  qx = fminf(fmaxf(qx, (float)c.lo[0] * B + .5f), (float)(c.hi[0] + 1) * B - .5f);
  qy = fminf(fmaxf(qy, (float)c.lo[1] * B + .5f), (float)(c.hi[1] + 1) * B - .5f);
  qz = fminf(fmaxf(qz, (float)c.lo[2] * B + .5f), (float)(c.hi[2] + 1) * B - .5f);
  float gx = qx - .5f, gy = qy - .5f, gz = qz - .5f;
  int x0 = (int)floorf(gx), y0 = (int)floorf(gy), z0 = (int)floorf(gz);
  float fx = gx - (float)x0, fy = gy - (float)y0, fz = gz - (float)z0;
  float v = 0.f;
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
    v += rawSmoke(P, R, c, x0 + dx, y0 + dy, z0 + dz) * w;
  }
  return v;
}
// smoothSmoke's [1,2,1]/4 density at a world cell: eight half-offset samples.
template <class Cursor>
FP_DEV float smoothedSmoke(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z) {
  float d = 0.f;
  for (int k = 0; k < 8; k++)
    d += smokeSample(P, R, c, (float)(x + (k & 1)), (float)(y + ((k >> 1) & 1)), (float)(z + (k >> 2)));
  return fmaxf(0.f, d * .125f);
}

// The coarse smoke grid (smoke_divisor d > 1): 2^P.smokeShift cells a brick side.
// The simulation's coarse density at a coarse cell: zero outside the box or without a slot.
template <class Cursor>
FP_DEV float rawCoarse(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z) {
  const int sh = P.smokeShift, m = (1 << sh) - 1;
  int s = slotAt(P, R, c, x >> sh, y >> sh, z >> sh);
  if (s < 0) return 0.f;
  return ldHalf(P.smk, (size_t)s * P.smokeCells + (((z & m) << sh | (y & m)) << sh | (x & m)), P.scalarHalf != 0);
}
// fireProField of the coarse density at `q` in coarse cells: clamped to the box, trilinear.
template <class Cursor>
FP_DEV float coarseSample(const SimParams& P, const FpRender& R, Cursor& c, float qx, float qy, float qz) {
  float S = (float)(1 << P.smokeShift);
  qx = fminf(fmaxf(qx, (float)c.lo[0] * S + .5f), (float)(c.hi[0] + 1) * S - .5f);
  qy = fminf(fmaxf(qy, (float)c.lo[1] * S + .5f), (float)(c.hi[1] + 1) * S - .5f);
  qz = fminf(fmaxf(qz, (float)c.lo[2] * S + .5f), (float)(c.hi[2] + 1) * S - .5f);
  float gx = qx - .5f, gy = qy - .5f, gz = qz - .5f;
  int x0 = (int)floorf(gx), y0 = (int)floorf(gy), z0 = (int)floorf(gz);
  float fx = gx - (float)x0, fy = gy - (float)y0, fz = gz - (float)z0;
  float v = 0.f;
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
    v += rawCoarse(P, R, c, x0 + dx, y0 + dy, z0 + dz) * w;
  }
  return v;
}
// smoothCoarseSmoke (lighting.wgsl:104-129): the [1,2,1]/4 density at a coarse cell.
template <class Cursor>
FP_DEV float smoothedCoarse(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z) {
  float d = 0.f;
  for (int k = 0; k < 8; k++)
    d += coarseSample(P, R, c, (float)(x + (k & 1)), (float)(y + ((k >> 1) & 1)), (float)(z + (k >> 2)));
  return fmaxf(0.f, d * .125f);
}
// The smoothed coarse density at a coarse cell: the pool in a brick with a slot, else what a
// sample based in a slotted brick reads from its apron (`apron`), else zero.
template <class Cursor>
FP_DEV float renderSmokeCell(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z, bool apron) {
  const int sh = P.smokeShift, m = (1 << sh) - 1;
  int s = slotAt(P, R, c, x >> sh, y >> sh, z >> sh);
  if (s >= 0) return R.renderSmoke[(size_t)s * P.smokeCells + (((z & m) << sh | (y & m)) << sh | (x & m))];
  if (!apron) return 0.f;
  if (s <= -2) return R.apronSmoke[(size_t)(-2 - s) * 3 * (m + 1) * (m + 1) + apronIndex(m + 1, x & m, y & m, z & m)];
  return smoothedCoarse(P, R, c, x, y, z);
}
// renderSmokeAt (volume-common.wgsl:74-78): fireProField of the smoothed coarse density at `q`
// in coarse cells.
template <class Cursor>
FP_DEV float renderSmokeAt(const SimParams& P, const FpRender& R, Cursor& c, float qx, float qy, float qz) {
  const int sh = P.smokeShift;
  float S = (float)(1 << sh);
  qx = fminf(fmaxf(qx, (float)c.lo[0] * S + .5f), (float)(c.hi[0] + 1) * S - .5f);
  qy = fminf(fmaxf(qy, (float)c.lo[1] * S + .5f), (float)(c.hi[1] + 1) * S - .5f);
  qz = fminf(fmaxf(qz, (float)c.lo[2] * S + .5f), (float)(c.hi[2] + 1) * S - .5f);
  float gx = qx - .5f, gy = qy - .5f, gz = qz - .5f;
  int x0 = (int)floorf(gx), y0 = (int)floorf(gy), z0 = (int)floorf(gz);
  float fx = gx - (float)x0, fy = gy - (float)y0, fz = gz - (float)z0;
  float v = 0.f;
  int slots[8];
  if (slots8(R, c, sh, x0, y0, z0, 1, slots)) {
    const int m = (1 << sh) - 1;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
      float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
      v += __ldg(&R.renderSmoke[(size_t)slots[k] * P.smokeCells +
                                ((((z0 + dz) & m) << sh | ((y0 + dy) & m)) << sh | ((x0 + dx) & m))]) * w;
    }
    return v;
  }
  bool based = slotAt(P, R, c, x0 >> sh, y0 >> sh, z0 >> sh) >= 0;
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
    v += renderSmokeCell(P, R, c, x0 + dx, y0 + dy, z0 + dz, based) * w;
  }
  return v;
}
// cachedSmokeCell (lighting.wgsl:133-156): the smoothed coarse density a conservative bound
// reads at coarse cell (x,y,z): the pool, else the apron a previous neighbour holds.
template <class Cursor>
FP_DEV float cachedSmokeCell(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z) {
  const int sh = P.smokeShift, m = (1 << sh) - 1;
  int bx = x >> sh, by = y >> sh, bz = z >> sh;
  int s = slotAt(P, R, c, bx, by, bz);
  if (s >= 0) return R.renderSmoke[(size_t)s * P.smokeCells + (((z & m) << sh | (y & m)) << sh | (x & m))];
  const int l[3] = {x & m, y & m, z & m};
  for (int k = 1; k < 8; k++) {
    if (((k & 1) && l[0] != 0) || ((k & 2) && l[1] != 0) || ((k & 4) && l[2] != 0)) continue;
    if (slotAt(P, R, c, bx - (k & 1), by - ((k >> 1) & 1), bz - ((k >> 2) & 1)) >= 0)
      return renderSmokeCell(P, R, c, x, y, z, true);
  }
  return 0.f;
}

// The render field at a world cell. A cell of a brick with a slot reads the pool. A cell in a
// brick without one reads as the apron of a sample based in a slotted brick would hold it
// (`apron`: the smoothed density, no heat, flame or fuel; all zero with coarse smoke, whose
// field apron holds no neighbour), else zero.
template <class Cursor>
FP_DEV float4 renderCell(const SimParams& P, const FpRender& R, Cursor& c, int x, int y, int z, bool apron) {
  int s = slotAt(P, R, c, x >> P.shift, y >> P.shift, z >> P.shift);
  if (s >= 0) return __ldg(&R.renderField[(size_t)s * P.N + localCell(P, x, y, z)]);
  if (!apron || P.smokeDiv > 1) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (s <= -2) {
    const int m = P.B - 1;
    return make_float4(R.apronField[(size_t)(-2 - s) * 3 * P.B * P.B + apronIndex(P.B, x & m, y & m, z & m)], 0.f, 0.f, 0.f);
  }
  return make_float4(smoothedSmoke(P, R, c, x, y, z), 0.f, 0.f, 0.f);
}
FP_DEV void add4(float4& a, const float4& b, float w) {
  a.x += b.x * w;
  a.y += b.y * w;
  a.z += b.z * w;
  a.w += b.w * w;
}
// The trilinear sample of the 2x2x2 block from cell (x0,y0,z0) when a cell of it has no slot or
// lies past the box: a lookup a cell. Out of line, so that the rare path costs the march and the
// lighting neither registers nor instruction-cache space.
template <class Cursor>
static __device__ __noinline__ float4 renderSampleFar(const SimParams& P, const FpRender& R, Cursor c, int x0, int y0,
                                                      int z0, float fx, float fy, float fz) {
  bool based = slotAt(P, R, c, x0 >> P.shift, y0 >> P.shift, z0 >> P.shift) >= 0;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
    add4(v, renderCell(P, R, c, x0 + dx, y0 + dy, z0 + dz, based), w);
  }
  return v;
}
// fireProField of the render field at `q` in cells (fireProSample, volume-bricks.wgsl).
template <class Cursor>
FP_DEV float4 renderSample(const SimParams& P, const FpRender& R, Cursor& c, float qx, float qy, float qz) {
  float B = (float)P.B;
  qx = fminf(fmaxf(qx, (float)c.lo[0] * B + .5f), (float)(c.hi[0] + 1) * B - .5f);
  qy = fminf(fmaxf(qy, (float)c.lo[1] * B + .5f), (float)(c.hi[1] + 1) * B - .5f);
  qz = fminf(fmaxf(qz, (float)c.lo[2] * B + .5f), (float)(c.hi[2] + 1) * B - .5f);
  float gx = qx - .5f, gy = qy - .5f, gz = qz - .5f;
  int x0 = (int)floorf(gx), y0 = (int)floorf(gy), z0 = (int)floorf(gz);
  float fx = gx - (float)x0, fy = gy - (float)y0, fz = gz - (float)z0;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  int slots[8];
  if (slots8(R, c, P.shift, x0, y0, z0, 1, slots)) {
    const unsigned sh = P.shift, m = P.B - 1;
    const unsigned lx[2] = {x0 & m, (x0 + 1) & m}, ly[2] = {(y0 & m) << sh, ((y0 + 1) & m) << sh},
                   lz[2] = {(z0 & m) << (2 * sh), ((z0 + 1) & m) << (2 * sh)};
    const unsigned N = P.N;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
      float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
      add4(v, __ldg(&R.renderField[(unsigned)slots[k] * N + (lx[dx] + ly[dy] + lz[dz])]), w);
    }
    return v;
  }
  return renderSampleFar(P, R, c, x0, y0, z0, fx, fy, fz);
}

// Two FP32 multiply-adds an instruction (fma.rn.f32x2): a render-field cell is two pairs.
struct Pair4 {
  unsigned long long a, b;
};
FP_DEV unsigned long long both(float w) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(w));
  return r;
}
FP_DEV void fma4(Pair4& v, const Pair4& t, unsigned long long w) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v.a) : "l"(t.a), "l"(w));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v.b) : "l"(t.b), "l"(w));
}
// The tensor-product sum of the NT^3 cells from (x0,y0,z0) with weights w[axis][tap], all in
// slotted bricks of the box (slots8's answer). x innermost, then y, then z.
template <int NT>
FP_DEV float4 tensorSample(const SimParams& P, const FpRender& R, const int* slots, int x0, int y0, int z0,
                           const float (*w)[4]) {
  const int sh = P.shift, m = P.B - 1, bx = x0 >> sh, by = y0 >> sh, bz = z0 >> sh;
  unsigned base[8];
#pragma unroll
  for (int k = 0; k < 8; k++) base[k] = (unsigned)slots[k] * (unsigned)P.N;
  const ulonglong2* F = reinterpret_cast<const ulonglong2*>(R.renderField);
  unsigned long long wx[NT];
  unsigned ox[NT];
  bool hx[NT];
#pragma unroll
  for (int i = 0; i < NT; i++) {
    wx[i] = both(w[0][i]);
    ox[i] = (unsigned)((x0 + i) & m);
    hx[i] = ((x0 + i) >> sh) != bx;
  }
  Pair4 v{0ull, 0ull};
  // A plane of the block at a time: its loads in flight together, and the code of one plane only
  // (the whole block unrolled cost the march a fifth of its issue slots in instruction misses).
#pragma unroll 1
  for (int k = 0; k < NT; k++) {
    const bool hz = ((z0 + k) >> sh) != bz;
    const unsigned lz = (unsigned)((z0 + k) & m) << (2 * sh);
    const unsigned b00 = hz ? base[4] : base[0], b10 = hz ? base[5] : base[1], b01 = hz ? base[6] : base[2],
                   b11 = hz ? base[7] : base[3];
    Pair4 plane{0ull, 0ull};
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const bool hy = ((y0 + j) >> sh) != by;
      const unsigned l = lz + ((unsigned)((y0 + j) & m) << sh), r0 = (hy ? b01 : b00) + l, r1 = (hy ? b11 : b10) + l;
      Pair4 row{0ull, 0ull};
#pragma unroll
      for (int i = 0; i < NT; i++) {
        const ulonglong2 q = __ldg(F + ((hx[i] ? r1 : r0) + ox[i]));
        fma4(row, Pair4{q.x, q.y}, wx[i]);
      }
      fma4(plane, row, both(w[1][j]));
    }
    fma4(v, plane, both(k == 0 ? w[2][0] : (k == 1 ? w[2][1] : (k == 2 ? w[2][2] : w[2][3]))));
  }
  float4 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v.a));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.z), "=f"(r.w) : "l"(v.b));
  return r;
}

// The B-spline as eight trilinear samples, when a cell of its block has no slot or lies past the
// box (each sample then decides by itself what the missing cells hold and where it clamps).
template <class Cursor>
static __device__ __noinline__ float4 reconstructFar(const SimParams& P, const FpRender& R, Cursor c, float px,
                                                     float py, float pz, int mode) {
  float pos[2][3], wt[2][3];
  float p[3] = {px, py, pz};
  for (int a = 0; a < 3; a++) {
    float g = p[a] - .5f;
    if (mode == 1) {
      float center = floorf(g + .5f), delta = g - center;
      float w0 = .5f * (.5f - delta) * (.5f - delta), w1 = .75f - delta * delta, w2 = .5f * (.5f + delta) * (.5f + delta);
      wt[0][a] = w0 + w1;
      wt[1][a] = w2;
      pos[0][a] = center - .5f + w1 / wt[0][a];
      pos[1][a] = center + 1.5f;
    } else {
      float base = floorf(g), q = g - floorf(g), inv = 1.f - q;
      float w0 = inv * inv * inv / 6.f, w1 = (3.f * q * q * q - 6.f * q * q + 4.f) / 6.f;
      float w2 = (-3.f * q * q * q + 3.f * q * q + 3.f * q + 1.f) / 6.f, w3 = q * q * q / 6.f;
      wt[0][a] = w0 + w1;
      wt[1][a] = w2 + w3;
      pos[0][a] = base - .5f + w1 / wt[0][a];
      pos[1][a] = base + 1.5f + w3 / wt[1][a];
    }
  }
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  // The reference's order: x outermost, then y, then z.
  for (int i = 0; i < 8; i++) {
    int ix = (i >> 2) & 1, iy = (i >> 1) & 1, iz = i & 1;
    add4(v, renderSample(P, R, c, pos[ix][0], pos[iy][1], pos[iz][2]), wt[ix][0] * wt[iy][1] * wt[iz][2]);
  }
  return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
}

// fireProReconstruct (volume-reconstruction.wgsl:5-95): 0 trilinear; 1 quadratic and 2 cubic
// B-splines. The reference takes eight trilinear samples, a sampler's filtering being free there.
// Here a sample is eight loads and as many lookups, and the eight touch just the 3^3 or 4^3 cells
// under the spline once each: with every one of them in a slotted brick of the box (the window then
// clamps nowhere) the same sum is taken over the cells directly, one vector load and two packed
// multiply-adds a cell.
template <class Cursor>
FP_DEV float4 reconstruct(const SimParams& P, const FpRender& R, Cursor& c, float px, float py, float pz, int mode) {
  if (mode == 0) return renderSample(P, R, c, px, py, pz);
  float w[3][4];
  int first[3];
  const float p[3] = {px, py, pz};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float g = p[a] - .5f;
    if (mode == 1) {
      const float center = floorf(g + .5f), delta = g - center;
      first[a] = (int)center - 1;
      w[a][0] = .5f * (.5f - delta) * (.5f - delta);
      w[a][1] = .75f - delta * delta;
      w[a][2] = .5f * (.5f + delta) * (.5f + delta);
      w[a][3] = 0.f;
    } else {
      const float base = floorf(g), q = g - base, inv = 1.f - q;
      first[a] = (int)base - 1;
      w[a][0] = inv * inv * inv / 6.f;
      w[a][1] = (3.f * q * q * q - 6.f * q * q + 4.f) / 6.f;
      w[a][2] = (-3.f * q * q * q + 3.f * q * q + 3.f * q + 1.f) / 6.f;
      w[a][3] = q * q * q / 6.f;
    }
  }
  int slots[8];
  // The quadratic's eight samples look at a fourth cell too, with weight zero: what it holds does
  // not matter, where the box clamps them does.
  if (!slots8(R, c, P.shift, first[0], first[1], first[2], 3, slots)) return reconstructFar(P, R, c, px, py, pz, mode);
  const float4 v = mode == 1 ? tensorSample<3>(P, R, slots, first[0], first[1], first[2], w)
                             : tensorSample<4>(P, R, slots, first[0], first[1], first[2], w);
  return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
}

// fireProExtinction and fireProEmission (fire-emission.wgsl:18-56).
FP_DEV float extinctionOf(const FpRender& R, const float4& f) {
  return fmaxf(0.f, f.x) * R.optical[0] + glowOf(f.z) * R.flameOpacity;
}
// What the fire's tint makes of the blackbody colour, the same for every sample.
struct Tint {
  float peak, saturation;
};
FP_DEV Tint tintOf(const FpRender& R) {
  Tint t;
  t.peak = fmaxf(R.fire[0], fmaxf(R.fire[1], R.fire[2]));
  t.saturation = 1.f - fminf(R.fire[0], fminf(R.fire[1], R.fire[2])) / fmaxf(t.peak, 1e-6f);
  return t;
}
FP_DEV float3 emissionOf(const FpRender& R, const Tint& tint, const float4& f) {
  if (R.optical[1] <= 0.f) return make_float3(0.f, 0.f, 0.f);
  float s = fmaxf(0.f, f.x) * R.optical[0], flame = glowOf(f.z) * R.flameOpacity;
  float3 source = make_float3((1.f - R.smoke[0]) * s * R.smoke[3] + flame, (1.f - R.smoke[1]) * s * R.smoke[3] + flame,
                              (1.f - R.smoke[2]) * s * R.smoke[3] + flame);
  if (source.x == 0.f && source.y == 0.f && source.z == 0.f) return make_float3(0.f, 0.f, 0.f);
  float heat = fmaxf(0.f, f.y);
  float kelvin = 800.f + heat / (heat + 2.f) * (R.fire[3] - 800.f);
  float u = fminf(fmaxf((kelvin - 500.f) / 9500.f, 0.f), 1.f) * (float)(FP_BLACKBODY_SIZE - 1);
  int i0 = (int)floorf(u);
  int i1 = min(i0 + 1, FP_BLACKBODY_SIZE - 1);
  float fr = u - (float)i0;
  float4 a = __ldg(&R.lut[i0]), b = __ldg(&R.lut[i1]);
  float4 spec = make_float4(mixf(a.x, b.x, fr), mixf(a.y, b.y, fr), mixf(a.z, b.z, fr), mixf(a.w, b.w, fr));
  float scale = exp2f(fminf(fmaxf(spec.w, -24.f), 10.f));
  float3 thermal = make_float3(spec.x * scale, spec.y * scale, spec.z * scale);
  const float tintPeak = tint.peak, saturation = tint.saturation;
  float peak = fmaxf(thermal.x, fmaxf(thermal.y, thermal.z));
  float k = R.optical[1];
  return make_float3(mixf(thermal.x * tintPeak, R.fire[0] * peak, saturation) * source.x * k,
                     mixf(thermal.y * tintPeak, R.fire[1] * peak, saturation) * source.y * k,
                     mixf(thermal.z * tintPeak, R.fire[2] * peak, saturation) * source.z * k);
}

// sampleWorld (volume-common.wgsl:33-43): the render field at world point p, zero outside
// the box.
template <class Cursor>
FP_DEV float4 sampleWorld(const SimParams& P, const FpRender& R, Cursor& c, float px, float py, float pz) {
  float size = (float)P.B * P.h;
  if (px < (float)c.lo[0] * size || py < (float)c.lo[1] * size || pz < (float)c.lo[2] * size ||
      px > (float)(c.hi[0] + 1) * size || py > (float)(c.hi[1] + 1) * size || pz > (float)(c.hi[2] + 1) * size)
    return make_float4(0.f, 0.f, 0.f, 0.f);
  float4 f = renderSample(P, R, c, px / P.h, py / P.h, pz / P.h);
  if (P.smokeDiv > 1) {
    const float r = 1.f / (float)P.smokeDiv;  // fine cells to coarse: a power of two, exact
    f.x = renderSmokeAt(P, R, c, px / P.h * r, py / P.h * r, pz / P.h * r);
  }
  return f;
}

// exitDistance (lighting.wgsl:248-255).
template <class Cursor>
FP_DEV float exitDistance(const SimParams& P, const Cursor& c, float px, float py, float pz, float dx, float dy,
                          float dz) {
  float size = (float)P.B * P.h;
  float p[3] = {px, py, pz}, d[3] = {dx, dy, dz}, m = 1e30f;
  for (int a = 0; a < 3; a++) {
    if (!(fabsf(d[a]) > 1e-6f)) continue;
    float edge = (d[a] > 0.f ? (float)(c.hi[a] + 1) : (float)c.lo[a]) * size;
    m = fminf(m, (edge - p[a]) / d[a]);
  }
  return fmaxf(0.f, m);
}

// integratedTransmission (volume-common.wgsl:47-53).
FP_DEV float integratedTransmission(float extinction, float distance, float attenuation) {
  float depth = extinction * distance;
  if (depth < .001f) return distance * (1.f - .5f * depth + depth * depth / 6.f);
  return (1.f - attenuation) / extinction;
}

// The glow's six rays.
FP_DEV float glowRay(int d, int axis) {
  const float sign = (d & 1) ? -1.f : 1.f;
  if (d < 2) return sign * (axis == 0 ? .36f : (axis == 1 ? .48f : -.8f));
  if (d < 4) return sign * (axis == 0 ? -.8f : (axis == 1 ? .6f : 0.f));
  return sign * (axis == 0 ? .48f : (axis == 1 ? .64f : .6f));
}
// incidentLight (lighting.wgsl:257-310): glow RGB and the sun's transmittance at p.
template <class Cursor>
FP_DEV float4 incidentLight(const SimParams& P, const FpRender& R, Cursor& c, float px, float py, float pz) {
  const Tint tint = tintOf(R);
  float4 local = sampleWorld(P, R, c, px, py, pz);
  if (local.x + glowOf(local.z) < 1e-5f) return make_float4(0.f, 0.f, 0.f, 1.f);
  float ln = sqrtf(R.light[0] * R.light[0] + R.light[1] * R.light[1] + R.light[2] * R.light[2]);
  float sx = R.light[0] / ln, sy = R.light[1] / ln, sz = R.light[2] / ln;
  int count = R.shadowSamples;
  float ds = exitDistance(P, c, px, py, pz, sx, sy, sz) / (float)count;
  float depth = 0.f;
  if (R.light[3] > 0.f) {
    for (int i = 0; i < count; i++) {
      float t = ((float)i + .5f) * ds;
      float4 f = sampleWorld(P, R, c, px + sx * t, py + sy * t, pz + sz * t);
      depth += (fmaxf(0.f, f.x) * R.optical[2] + glowOf(f.z) * R.flameOpacity) * ds;
      if (depth > 9.f) break;
    }
  }
  float3 glow = make_float3(0.f, 0.f, 0.f);
  if (R.optical[1] > 0.f && local.x > 1e-5f) {
    for (int d = 0; d < 6; d++) {
      float t = 0.f, interval = .075f, transmission = 1.f;
      for (int s = 0; s < 6; s++) {
        float q = t + interval * .5f;
        float4 f = sampleWorld(P, R, c, px + glowRay(d, 0) * q, py + glowRay(d, 1) * q, pz + glowRay(d, 2) * q);
        float ext = extinctionOf(R, f);
        float att = expf(-ext * interval);
        float3 e = emissionOf(R, tint, f);
        float w = transmission * integratedTransmission(ext, interval, att) / 6.f;
        glow.x += e.x * w;
        glow.y += e.y * w;
        glow.z += e.z * w;
        transmission *= att;
        t += interval;
        interval *= 1.65f;
      }
    }
  }
  return make_float4(glow.x, glow.y, glow.z, expf(-depth));
}

// The brick of computing brick `i` inside a box, that box made the current one, with its
// slot; false when no box holds it.
template <class Cursor>
FP_DEV bool boxBrick(const SimParams& P, const FpRender& R, Cursor& c, uint32_t i, int& bx, int& by, int& bz,
                     int& slot) {
  uint32_t id = P.active[i];
  if (!homeOk(P, id)) return false;  // the bounds-checked build only
  int4 t = __ldg(&P.tileRec[id >> 6]);
  int l = id & 63;
  bx = t.x * 4 + (l & 3);
  by = t.y * 4 + ((l >> 2) & 3);
  bz = t.z * 4 + (l >> 4);
  int k = 0;
  for (; k < R.boxCount; k++) {
    const int* b = R.boxes + FP_BOX_INTS * k;
    if (bx >= b[0] && bx <= b[3] && by >= b[1] && by <= b[4] && bz >= b[2] && bz <= b[5]) break;
  }
  if (k == R.boxCount) return false;
  useBox(R, c, k);
  slot = slotAt(P, R, c, bx, by, bz);
  return slot >= 0;
}

// The boxes' brick tables: a hash lookup a brick of a box, once a render, in place of one at every
// brick a ray or a light sample enters.
__global__ void __launch_bounds__(256) k_render_pages(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  if (R.apronCap && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *R.apronCount = 0;
  for (int k = blockIdx.y; k < R.boxCount; k += gridDim.y) {
    const int* b = R.boxes + FP_BOX_INTS * k;
    const int nx = b[3] - b[0] + 1, ny = b[4] - b[1] + 1, nz = b[5] - b[2] + 1, total = nx * ny * nz;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
      R.pages[b[6] + i] = hashedSlot(P, b[0] + i % nx, b[1] + i / nx % ny, b[2] + i / (nx * ny));
  }
}
// The apron bricks of the boxes, numbered in the order they are met (what one holds depends on its
// place alone, not on its number). The tables are written while they are read: only from -1 to
// less, and a neighbour's sign is all that is read.
__global__ void __launch_bounds__(256) k_render_aprons(const __grid_constant__ FpRender R) {
  const volatile int* pages = R.pages;
  for (int k = blockIdx.y; k < R.boxCount; k += gridDim.y) {
    const int* b = R.boxes + FP_BOX_INTS * k;
    const int nx = b[3] - b[0] + 1, ny = b[4] - b[1] + 1, nz = b[5] - b[2] + 1, total = nx * ny * nz;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
      if (pages[b[6] + i] != -1) continue;
      const int x = i % nx, y = i / nx % ny, z = i / (nx * ny);
      bool after = false;
#pragma unroll
      for (int q = 1; q < 8; q++) {
        const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
        if (x >= dx && y >= dy && z >= dz && pages[b[6] + i - dx - dy * nx - dz * nx * ny] >= 0) after = true;
      }
      if (!after) continue;
      const int g = atomicAdd(R.apronCount, 1);
      if (g >= R.apronCap) continue;
      R.apronBricks[g] = make_int4(b[0] + x, b[1] + y, b[2] + z, k);
      R.pages[b[6] + i] = -2 - g;
    }
  }
}
FP_DEV uint32_t apronTotal(const FpRender& R) { return R.apronCap ? (uint32_t)min(*R.apronCount, R.apronCap) : 0u; }

// The [1,2,1]/4 density of a block of side `bs` cells (8, or a coarse brick's 2 or 4) whose first
// cell is (ox,oy,oz), on a lattice of 2^sh cells a brick: smoothSmoke's and smoothCoarseSmoke's
// eight half-offset samples a cell share their corners, so the block's (bs + 2)^3 cells are staged
// once, the (bs + 1)^3 corner samples taken from the stage, and each cell's eight of them summed.
// The sums and their order are smoothedSmoke's; `raw` reads a cell (zero outside the box or
// without a slot) and `put` takes cell k of the block and its density. Every thread of the CTA
// calls it.
// What bounds it: reading a cell through the brick tables cost 64 lookups and loads a cell when
// every cell took its own eight samples (427 us on 3.7k bricks of 8^3, 216 us on 1.8k).
struct SmoothStage {
  float cells[1000], corners[729];
};
template <class Cursor, class Raw, class Put>
FP_DEV void smoothBlock(const Cursor& c, SmoothStage& st, int sh, int ox, int oy, int oz, int bs, Raw raw, Put put) {
  const int S = bs + 2, C = bs + 1;
  for (int i = threadIdx.x; i < S * S * S; i += RTHREADS)
    st.cells[i] = raw(ox - 1 + i % S, oy - 1 + i / S % S, oz - 1 + i / (S * S));
  __syncthreads();
  // Corner i of an axis lies between cells i - 1 and i of the block; at the box's own faces the
  // sample clamps to the centre of the cell inside it.
  const int o[3] = {ox, oy, oz};
  for (int i = threadIdx.x; i < C * C * C; i += RTHREADS) {
    const int q[3] = {i % C, i / C % C, i / (C * C)};
    int f0[3];
    float fr[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const bool low = o[a] + q[a] == (c.lo[a] << sh), high = o[a] + q[a] == ((c.hi[a] + 1) << sh);
      f0[a] = low ? q[a] + 1 : q[a];  // the staged place of the sample's first cell
      fr[a] = low || high ? 0.f : .5f;
    }
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
      const float w = (dx ? fr[0] : 1.f - fr[0]) * (dy ? fr[1] : 1.f - fr[1]) * (dz ? fr[2] : 1.f - fr[2]);
      if (w != 0.f) v += st.cells[((f0[2] + dz) * S + f0[1] + dy) * S + f0[0] + dx] * w;
    }
    st.corners[i] = v;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < bs * bs * bs; k += RTHREADS) {
    const int x = k % bs, y = k / bs % bs, z = k / (bs * bs);
    float d = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) d += st.corners[((z + (j >> 2)) * C + y + ((j >> 1) & 1)) * C + x + (j & 1)];
    put(k, fmaxf(0.f, d * .125f));
  }
}

// smoothSmoke: the render field of each boxed brick, the smoothed density with heat, lifetime and
// fuel as they are; the coarse density smoothed on its own lattice; the aprons of both; and each
// 2x2x2 cells' maxima for the occupancy. A CTA an 8^3 block, so that bricks of 16^3 and 32^3 spread
// over the chip too.
template <class Cursor>
__global__ void __launch_bounds__(RTHREADS) k_render_field(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  __shared__ SmoothStage st;
  __shared__ float2 cellMax[512];
  const uint32_t total = P.counters->active, aprons = apronTotal(R);
  const bool half = P.scalarHalf != 0, coarse = P.smokeDiv > 1;
  const int per = P.B / 8, blocks = per * per * per;
  const int ssh = P.smokeShift, SB = 1 << ssh, sbs = SB < 8 ? SB : 8, sper = coarse ? SB / sbs : 0, sblocks = sper * sper * sper;
  for (uint32_t item = blockIdx.x; item < (total + aprons) * (uint32_t)blocks; item += gridDim.x) {
    const uint32_t i = item / blocks;
    const int b = item % blocks, ox = b % per * 8, oy = b / per % per * 8, oz = b / (per * per) * 8;
    const int sx = coarse ? b % sper * sbs : 0, sy = coarse ? b / sper % sper * sbs : 0,
              sz = coarse ? b / (sper * sper) * sbs : 0;  // the coarse block b, when there are that many
    Cursor c = noBox<Cursor>();
    auto fine = [&](int x, int y, int z) { return rawSmoke(P, R, c, x, y, z); };
    auto thin = [&](int x, int y, int z) { return rawCoarse(P, R, c, x, y, z); };
    __syncthreads();  // the previous block's stage has been read
    if (i >= total) {
      // An apron brick: its cells on the low faces.
      const uint32_t g = i - total;
      const int4 q = R.apronBricks[g];
      useBox(R, c, q.w);
      const int side = coarse ? SB : P.B, bs = coarse ? sbs : 8, cx = coarse ? sx : ox, cy = coarse ? sy : oy,
                cz = coarse ? sz : oz;
      if ((coarse && b >= sblocks) || (cx > 0 && cy > 0 && cz > 0)) continue;  // the same for the whole CTA
      float* out = (coarse ? R.apronSmoke : R.apronField) + (size_t)g * 3 * side * side;
      auto put = [&](int k, float d) {
        const int lx = cx + k % bs, ly = cy + k / bs % bs, lz = cz + k / (bs * bs);
        if (lx == 0 || ly == 0 || lz == 0) out[apronIndex(side, lx, ly, lz)] = d;
      };
      if (coarse)
        smoothBlock(c, st, ssh, q.x * side + cx, q.y * side + cy, q.z * side + cz, bs, thin, put);
      else
        smoothBlock(c, st, P.shift, q.x * side + cx, q.y * side + cy, q.z * side + cz, bs, fine, put);
      continue;
    }
    int bx, by, bz, slot;
    if (!boxBrick(P, R, c, i, bx, by, bz, slot)) continue;  // the same for the whole CTA
    auto put = [&](int k, float d) {
      const int cell = (((oz + (k >> 6)) << P.shift) + oy + ((k >> 3) & 7)) * P.B + ox + (k & 7);
      const size_t o = (size_t)slot * 4 * P.N + cell;
      const float4 f = make_float4(d, ldHalf(P.fld, o + P.N, half), ldHalf(P.fld, o + 2 * P.N, half),
                                   ldHalf(P.fld, o + 3 * P.N, half));
      R.renderField[(size_t)slot * P.N + cell] = f;
      const float glow = glowOf(f.z);
      cellMax[k] = make_float2(glow, (coarse ? 0.f : f.x) + glow);
    };
    if (coarse) {
      for (int k = threadIdx.x; k < 512; k += RTHREADS) {
        const int cell = (((oz + (k >> 6)) << P.shift) + oy + ((k >> 3) & 7)) * P.B + ox + (k & 7);
        put(k, ldHalf(P.fld, (size_t)slot * 4 * P.N + cell, half));
      }
      if (b < sblocks)
        smoothBlock(c, st, ssh, bx * SB + sx, by * SB + sy, bz * SB + sz, sbs, thin, [&](int k, float d) {
          const int x = sx + k % sbs, y = sy + k / sbs % sbs, z = sz + k / (sbs * sbs);
          R.renderSmoke[(size_t)slot * P.smokeCells + ((((z << ssh) | y) << ssh) | x)] = d;
        });
    } else {
      smoothBlock(c, st, P.shift, bx * P.B + ox, by * P.B + oy, bz * P.B + oz, 8, fine, put);
    }
    __syncthreads();
    if (R.units && threadIdx.x < 64) {
      const int u = threadIdx.x, first = ((u >> 4) * 2 * 8 + ((u >> 2) & 3) * 2) * 8 + (u & 3) * 2;
      float2 m = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const float2 v = cellMax[first + ((k >> 2) * 8 + ((k >> 1) & 1)) * 8 + (k & 1)];
        m.x = fmaxf(m.x, v.x);
        m.y = fmaxf(m.y, v.y);
      }
      R.units[((size_t)slot * blocks + b) * 64 + u] = m;
    }
  }
}

// buildOccupancy (lighting.wgsl:149-244), a warp an 8^3 block: what is visible in the block and two
// cells around it, from the maxima of 2x2x2 cells (216 of them; each lies in one brick).
// UNITS: those maxima are there; else they are taken here, each some 27 times over.
template <class Cursor, bool UNITS>
__global__ void __launch_bounds__(RTHREADS) k_render_occupancy(const SimParams* __restrict__ Pp,
                                                               const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  const uint32_t total = P.counters->active;
  const int per = P.B / 8, blocks = per * per * per, lane = threadIdx.x & 31;
  const bool coarse = P.smokeDiv > 1;
  for (uint32_t item = blockIdx.x * (RTHREADS / 32) + (threadIdx.x >> 5); item < total * (uint32_t)blocks;
       item += gridDim.x * (RTHREADS / 32)) {
    Cursor c = noBox<Cursor>();
    int bx, by, bz, slot;
    if (!boxBrick(P, R, c, item / blocks, bx, by, bz, slot)) continue;  // the same for the whole warp
    const int b = item % blocks;
    const int ox = bx * P.B + b % per * 8 - 2, oy = by * P.B + b / per % per * 8 - 2, oz = bz * P.B + b / (per * per) * 8 - 2;
    float glow = 0.f, seen = 0.f;
#pragma unroll
    for (int u = lane; u < 216; u += 32) {
      const int ux = ox + (u % 6) * 2, uy = oy + ((u / 6) % 6) * 2, uz = oz + (u / 36) * 2, m = P.B - 1;
      const int s = slotAt(P, R, c, ux >> P.shift, uy >> P.shift, uz >> P.shift);
      if (s < 0) continue;
      const int block = (((uz & m) >> 3) * per + ((uy & m) >> 3)) * per + ((ux & m) >> 3);
      const int unit = (((uz & 7) >> 1) * 4 + ((uy & 7) >> 1)) * 4 + ((ux & 7) >> 1);
      if constexpr (UNITS) {
        const float2 v = __ldg(&R.units[((size_t)s * blocks + block) * 64 + unit]);
        glow = fmaxf(glow, v.x);
        seen = fmaxf(seen, v.y);
      } else {
        for (int k = 0; k < 8; k++) {
          const int cell = localCell(P, ux + (k & 1), uy + ((k >> 1) & 1), uz + (k >> 2));
          const float4 f = __ldg(&R.renderField[(size_t)s * P.N + cell]);
          const float g = glowOf(f.z);
          glow = fmaxf(glow, g);
          seen = fmaxf(seen, (coarse ? 0.f : f.x) + g);
        }
      }
    }
    float smoke = 0.f;
    if (coarse) {
      // Every trilinear donor of coarse density in the block and halo (lighting.wgsl:222-238).
      const int d = P.smokeDiv, S = 1 << P.smokeShift;
      const float ratio = (float)d;
      int lo[3], size[3], boxLo[3], boxHi[3];
      const int o[3] = {ox, oy, oz};
#pragma unroll
      for (int a = 0; a < 3; a++) {
        lo[a] = (int)floorf((float)o[a] / ratio - .5f);
        size[a] = (int)floorf((float)(o[a] + 12) / ratio - .5f) + 2 - lo[a];
        boxLo[a] = c.lo[a] * S;
        boxHi[a] = (c.hi[a] + 1) * S - 1;
      }
      for (int q = lane; q < size[0] * size[1] * size[2]; q += 32) {
        int cq[3] = {lo[0] + q % size[0], lo[1] + (q / size[0]) % size[1], lo[2] + q / (size[0] * size[1])};
#pragma unroll
        for (int a = 0; a < 3; a++) cq[a] = min(max(cq[a], boxLo[a]), boxHi[a]);
        smoke = fmaxf(smoke, cachedSmokeCell(P, R, c, cq[0], cq[1], cq[2]));
      }
    }
    // Nonnegative floats order as their bits.
    glow = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(glow)));
    seen = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(seen)));
    if (coarse) smoke = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(smoke)));
    if (lane == 0)
      R.occupancy[(size_t)slot * blocks + b] =
          (uint8_t)((glow > .002f ? 1 : 0) | (seen > .002f || (coarse && smoke + glow > .002f) ? 2 : 0));
  }
}

// buildLighting of each boxed brick and of the aprons, LIGHT_TEXELS texels of a brick a CTA. An
// incident light (incidentLight) is a sample where it stands, up to 256 samples towards the sun and
// six rays of six samples, each at a place known beforehand: the CTA takes the texels' samples as
// one flat list, a thread each, into shared memory; then four lanes a texel add them up in the
// serial order, one the sun's depth (with its early stop) and one each colour of the glow.
// All the sun's samples are taken, those too past the depth at which the sum then stops: a small image
// of 2.4k bricks takes 228 us with 16 samples a texel and 355 with 256 (in smoke fifty times as dense 346),
// where a warp a texel that stopped after the 32 in which it got there took 1.9 and 2.5 to 2.7 ms.
// A warp a texel left 26 lanes idle while six walked the rays: 1.9 -> 0.43 ms on the default
// grid's 640 bricks of 64 texels, 0.66 -> 0.21 ms on 3.7k bricks of 8.
constexpr int LIGHT_TEXELS = 16, GLOW_SAMPLES = 36, SUN_SAMPLES = 256;
struct LightStage {
  float sun[LIGHT_TEXELS][SUN_SAMPLES];
  float glow[LIGHT_TEXELS][5][GLOW_SAMPLES];  // emission RGB, the integrated transmission, the attenuation
  float4 at[LIGHT_TEXELS];                    // the lit texels: position, the sun samples' spacing
  float4* out[LIGHT_TEXELS];
  int glows[LIGHT_TEXELS];
  int count;
};
template <class Cursor>
__global__ void __launch_bounds__(RTHREADS) k_render_light(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  __shared__ LightStage st;
  const uint32_t total = P.counters->active, aprons = apronTotal(R);
  const int L = 1 << R.lightShift, L3 = L * L * L, planes = 3 * L * L;
  const uint32_t chunks = (L3 + LIGHT_TEXELS - 1) / LIGHT_TEXELS, apronChunks = (planes + LIGHT_TEXELS - 1) / LIGHT_TEXELS;
  const float texel = P.h * (float)(P.B >> R.lightShift);
  const Tint tint = tintOf(R);
  const float ln = sqrtf(R.light[0] * R.light[0] + R.light[1] * R.light[1] + R.light[2] * R.light[2]);
  const float sx = R.light[0] / ln, sy = R.light[1] / ln, sz = R.light[2] / ln;
  const int count = R.light[3] > 0.f ? R.shadowSamples : 0, perTexel = count + (R.optical[1] > 0.f ? GLOW_SAMPLES : 0);
  for (uint32_t item = blockIdx.x; item < total * chunks + aprons * apronChunks; item += gridDim.x) {
    Cursor c = noBox<Cursor>();
    int bx, by, bz, slot = 0;
    unsigned before = 0;
    const bool apron = item >= total * chunks;
    const uint32_t brick = apron ? (item - total * chunks) / apronChunks : item / chunks;
    const int first = (int)(apron ? (item - total * chunks) % apronChunks : item % chunks) * LIGHT_TEXELS;
    if (apron) {
      const int4 q = R.apronBricks[brick];
      useBox(R, c, q.w);
      bx = q.x;
      by = q.y;
      bz = q.z;
      before = slottedBefore(P, R, c, bx, by, bz);
    } else if (!boxBrick(P, R, c, brick, bx, by, bz, slot)) {
      continue;  // the same for the whole CTA
    }
    // The texels that anything is at: the others see the open sun and no glow.
    if (threadIdx.x < 32) {
      const int k = first + (int)threadIdx.x;
      bool lit = false;
      float4 at = make_float4(0.f, 0.f, 0.f, 0.f), local = at;
      float4* out = nullptr;
      if (threadIdx.x < LIGHT_TEXELS && k < (apron ? planes : L3)) {
        int lx = k % L, ly = (k / L) % L, lz = k / (L * L);
        if (!apron || apronCell(L, k, before, lx, ly, lz)) {
          out = apron ? R.apronLight + (size_t)brick * planes + k : R.lighting + (size_t)slot * L3 + k;
          at = make_float4(((float)(bx * L + lx) + .5f) * texel, ((float)(by * L + ly) + .5f) * texel,
                           ((float)(bz * L + lz) + .5f) * texel, 0.f);
          local = sampleWorld(P, R, c, at.x, at.y, at.z);
          lit = !(local.x + glowOf(local.z) < 1e-5f);
          if (!lit) *out = make_float4(0.f, 0.f, 0.f, 1.f);
        }
      }
      const unsigned mask = __ballot_sync(0xffffffffu, lit);
      if (lit) {
        const int j = __popc(mask & ((1u << threadIdx.x) - 1u));
        at.w = exitDistance(P, c, at.x, at.y, at.z, sx, sy, sz) / (float)R.shadowSamples;
        st.at[j] = at;
        st.out[j] = out;
        st.glows[j] = R.optical[1] > 0.f && local.x > 1e-5f;
      }
      if (threadIdx.x == 0) st.count = __popc(mask);
    }
    __syncthreads();
    const int n = st.count;
    for (int q = threadIdx.x; q < n * perTexel; q += RTHREADS) {
      const int j = q / perTexel, i = q - j * perTexel;
      const float4 at = st.at[j];
      if (i < count) {
        const float t = ((float)i + .5f) * at.w;
        const float4 f = sampleWorld(P, R, c, at.x + sx * t, at.y + sy * t, at.z + sz * t);
        st.sun[j][i] = (fmaxf(0.f, f.x) * R.optical[2] + glowOf(f.z) * R.flameOpacity) * at.w;
      } else if (st.glows[j]) {
        const int s = i - count, d = s / 6, k = s - d * 6;
        float t = 0.f, interval = .075f;
        for (int e = 0; e < k; e++) {
          t += interval;
          interval *= 1.65f;
        }
        const float p = t + interval * .5f;
        const float4 f = sampleWorld(P, R, c, at.x + glowRay(d, 0) * p, at.y + glowRay(d, 1) * p, at.z + glowRay(d, 2) * p);
        const float ext = extinctionOf(R, f), att = expf(-ext * interval);
        const float3 e = emissionOf(R, tint, f);
        st.glow[j][0][s] = e.x;
        st.glow[j][1][s] = e.y;
        st.glow[j][2][s] = e.z;
        st.glow[j][3][s] = integratedTransmission(ext, interval, att);
        st.glow[j][4][s] = att;
      }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n * 4; q += RTHREADS) {
      const int j = q >> 2, role = q & 3;
      float v = 0.f;
      if (role == 3) {
        float depth = 0.f;
        for (int i = 0; i < count; i++) {
          depth += st.sun[j][i];
          if (depth > 9.f) break;
        }
        v = expf(-depth);
      } else if (st.glows[j]) {
        for (int d = 0; d < 6; d++) {
          float transmission = 1.f;
#pragma unroll
          for (int k = 0; k < 6; k++) {
            const int s = d * 6 + k;
            v += st.glow[j][role][s] * (transmission * st.glow[j][3][s] / 6.f);
            transmission *= st.glow[j][4][s];
          }
        }
      }
      reinterpret_cast<float*>(st.out[j])[role] = v;
    }
    __syncthreads();  // the stage is read before the next texels' samples
  }
}

// The lighting sample whose texels' bricks are not all slotted: out of line, rare.
template <class Cursor>
static __device__ __noinline__ float4 lightSampleFar(const SimParams& P, const FpRender& R, Cursor c, int x0, int y0,
                                                     int z0, float fx, float fy, float fz) {
  const int L = 1 << R.lightShift, L3 = L * L * L;
  const float texel = P.h * (float)(P.B >> R.lightShift);
  if (slotAt(P, R, c, x0 >> R.lightShift, y0 >> R.lightShift, z0 >> R.lightShift) < 0)
    return make_float4(0.f, 0.f, 0.f, 1.f);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    int x = x0 + dx, y = y0 + dy, z = z0 + dz;
    float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
    int s = slotAt(P, R, c, x >> R.lightShift, y >> R.lightShift, z >> R.lightShift);
    float4 t;
    if (s >= 0) {
      const int m = L - 1;
      t = __ldg(&R.lighting[(size_t)s * L3 + (((z & m) * L + (y & m)) * L + (x & m))]);
    } else if (s <= -2) {
      const int m = L - 1;
      t = __ldg(&R.apronLight[(size_t)(-2 - s) * 3 * L * L + apronIndex(L, x & m, y & m, z & m)]);
    } else {  // the apron of a neighbour without a slot: lit where it stands
      t = incidentLight(P, R, c, ((float)x + .5f) * texel, ((float)y + .5f) * texel, ((float)z + .5f) * texel);
    }
    add4(v, t, w);
  }
  return v;
}
// fireProLight (volume-bricks.wgsl:158-178) at `q` in lighting texels.
template <class Cursor>
FP_DEV float4 lightSample(const SimParams& P, const FpRender& R, Cursor& c, float qx, float qy, float qz) {
  const int L = 1 << R.lightShift;
  qx = fminf(fmaxf(qx, (float)c.lo[0] * L + .5f), (float)(c.hi[0] + 1) * L - .5f);
  qy = fminf(fmaxf(qy, (float)c.lo[1] * L + .5f), (float)(c.hi[1] + 1) * L - .5f);
  qz = fminf(fmaxf(qz, (float)c.lo[2] * L + .5f), (float)(c.hi[2] + 1) * L - .5f);
  float gx = qx - .5f, gy = qy - .5f, gz = qz - .5f;
  int x0 = (int)floorf(gx), y0 = (int)floorf(gy), z0 = (int)floorf(gz);
  float fx = gx - (float)x0, fy = gy - (float)y0, fz = gz - (float)z0;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  int slots[8];
  if (slots8(R, c, R.lightShift, x0, y0, z0, 1, slots)) {
    const unsigned sh = R.lightShift, m = (1u << sh) - 1u;
    const unsigned lx[2] = {x0 & m, (x0 + 1) & m}, ly[2] = {(y0 & m) << sh, ((y0 + 1) & m) << sh},
                   lz[2] = {(z0 & m) << (2 * sh), ((z0 + 1) & m) << (2 * sh)};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
      float w = (dx ? fx : 1.f - fx) * (dy ? fy : 1.f - fy) * (dz ? fz : 1.f - fz);
      add4(v, __ldg(&R.lighting[((unsigned)slots[k] << (3 * sh)) + (lx[dx] + ly[dy] + lz[dz])]), w);
    }
    return v;
  }
  return lightSampleFar(P, R, c, x0, y0, z0, fx, fy, fz);
}

// fireProJitter (volume-march.wgsl:94-102).
FP_DEV float jitterOf(uint32_t px, uint32_t py, float time) {
  uint32_t s0 = px * 1664525u + 1013904223u, s1 = py * 1664525u + 1013904223u,
           s2 = (uint32_t)(time * 60.f) * 1664525u + 1013904223u;
  s0 += s1 * s2;
  s1 += s2 * s0;
  s2 += s0 * s1;
  s0 ^= s0 >> 16u;
  s1 ^= s1 >> 16u;
  s2 ^= s2 >> 16u;
  s0 += s1 * s2;
  return (float)(s0 >> 8u) / 16777216.f;
}

// A pixel's march (fireProSceneVolume with fireProMarch), a thread a pixel.
// A camera ray through the boxes (fireProRay, fireProSpan) and what its march keeps fixed.
struct Ray {
  float ro[3], rd[3];
  float lo, hi;  // the first box entry and the last exit
  float stepSize, jitter, direct;  // direct: the sun's factor (fireProDirect over sceneLight)
  float perSafe[3], perStep;       // 1 / safeAxis(rd), 1 / stepSize
};
FP_DEV float safeAxis(float d) { return fabsf(d) > 1e-6f ? d : 1e-6f; }
// fireProHit: where the ray enters and leaves box k (entry after exit when it misses).
FP_DEV float2 boxHit(const FpRender& R, const Ray& r, int k, float brickSize) {
  const int* b = R.boxes + FP_BOX_INTS * k;
  float lo = 0.f, hi = 1e30f;
  for (int a = 0; a < 3; a++) {
    float ta = ((float)b[a] * brickSize - r.ro[a]) / safeAxis(r.rd[a]);
    float tb = ((float)(b[3 + a] + 1) * brickSize - r.ro[a]) / safeAxis(r.rd[a]);
    lo = fmaxf(lo, fminf(ta, tb));
    hi = fminf(hi, fmaxf(ta, tb));
  }
  return make_float2(lo, hi);
}
// The ray of viewport point (ux, uy) in [0,1]^2, its span through the boxes and step; false
// when it misses them all.
FP_DEV bool rayOf(const SimParams& P, const FpRender& R, float ux, float uy, Ray& r) {
  float cx = ux * 2.f - 1.f, cy = 1.f - uy * 2.f;
  const float* M = R.ivp;
  float nh[4], fh[4];
  for (int k = 0; k < 4; k++) {
    nh[k] = M[k] * cx + M[4 + k] * cy + M[8 + k] * 0.f + M[12 + k];
    fh[k] = M[k] * cx + M[4 + k] * cy + M[8 + k] * .99999f + M[12 + k];
  }
  for (int a = 0; a < 3; a++) {
    r.ro[a] = nh[a] / nh[3];
    r.rd[a] = fh[a] / fh[3] - r.ro[a];
  }
  float rl = sqrtf(r.rd[0] * r.rd[0] + r.rd[1] * r.rd[1] + r.rd[2] * r.rd[2]);
  for (int a = 0; a < 3; a++) r.rd[a] /= rl;
  const float brickSize = P.h * (float)P.B;
  for (int a = 0; a < 3; a++) r.perSafe[a] = 1.f / safeAxis(r.rd[a]);
  // fireProSpan: the first entry, the last exit and the length inside every box.
  r.lo = 1e30f;
  r.hi = 0.f;
  float length = 0.f;
  for (int k = 0; k < R.boxCount; k++) {
    float2 hit = boxHit(R, r, k, brickSize);
    if (hit.y > hit.x) {
      r.lo = fminf(r.lo, hit.x);
      r.hi = fmaxf(r.hi, hit.y);
      length += hit.y - hit.x;
    }
  }
  if (!(r.hi > r.lo)) return false;
  r.stepSize = fmaxf(P.h * .5f, length / (float)R.raySteps);
  r.perStep = 1.f / r.stepSize;
  // fireProDirect
  float ln = sqrtf(R.light[0] * R.light[0] + R.light[1] * R.light[1] + R.light[2] * R.light[2]);
  float g = R.optical[3];
  float mu = (r.rd[0] * R.light[0] + r.rd[1] * R.light[1] + r.rd[2] * R.light[2]) / ln;
  float phase = (1.f - g * g) / powf(fmaxf(.05f, 1.f + g * g - 2.f * g * mu), 1.5f);
  r.direct = R.light[3] * (.35f + phase * .3f);
  return true;
}

// fireProEnter (fireProNext): the box the ray is in at t, or the next one it enters, becomes the
// current one with its exit, and t moves to its entry; false past the last box. Boxes never
// overlap, so of the boxes the ray has not left, the one it enters first is the one.
template <class Cursor>
FP_DEV bool enterBox(const SimParams& P, const FpRender& R, const Ray& r, float& t, float& exit, Cursor& c) {
  const float brickSize = P.h * (float)P.B;
  float entry = 1e30f, out = 0.f;
  int best = -1;
  for (int k = 0; k < R.boxCount; k++) {
    float2 hit = boxHit(R, r, k, brickSize);
    if (hit.y > hit.x && hit.y > t && hit.x < entry) {
      entry = hit.x;
      out = hit.y;
      best = k;
    }
  }
  if (best < 0) return false;
  useBox(R, c, best);
  exit = out;
  t = fmaxf(t, entry);
  return true;
}

// One sample of fireProMarch (volume-march.wgsl:178-268) at t, ds long, in the current box (which
// the ray leaves at `exit`).
struct Sample {
  bool lit;        // its block may hold something visible; else the ray goes on at `next`
  float next;      // past an empty block: whole steps beyond it, up to the exit
  float cell[3];   // the sample point in field cells
  int filter;      // the reconstruction filter of its block
};
template <class Cursor>
FP_DEV Sample sampleAt(const SimParams& P, const FpRender& R, Cursor& c, const Ray& r, float t, float ds, float exit) {
  Sample s;
  float tt = t + r.jitter * ds;
  float p[3] = {r.ro[0] + r.rd[0] * tt, r.ro[1] + r.rd[1] * tt, r.ro[2] + r.rd[2] * tt};
  int ci[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    s.cell[a] = p[a] / P.h;  // divided: which block a sample on its face falls in is a decision
    ci[a] = (int)floorf(s.cell[a]);
  }
  int slot = slotAt(P, R, c, ci[0] >> P.shift, ci[1] >> P.shift, ci[2] >> P.shift);
  int shift = P.shift;  // log2 cells of what is empty together: the brick, or the 8-cell block
  int flags = 0;
  if (slot >= 0) {  // fireProOccupancy: the sample's 8-cell block of the brick
    const int per = P.shift - 3, m = (1 << per) - 1;
    const int block = (((((ci[2] >> 3) & m) << per) | ((ci[1] >> 3) & m)) << per) | ((ci[0] >> 3) & m);
    flags = __ldg(&R.occupancy[((size_t)slot << (3 * per)) + block]);
    shift = 3;
  }
  s.lit = (flags & 2) != 0;
  s.filter = (flags & 1) ? R.filter : 0;
  s.next = t;
  if (!s.lit) {
    // Skip whole steps past the empty block, keeping the lattice. The count of steps is a decision
    // too: from reciprocals, unless it is near a whole number.
    float away[3], dist = 1e30f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int edge = ((ci[a] >> shift) + (r.rd[a] > 0.f ? 1 : 0)) << shift;
      away[a] = (float)edge * P.h - p[a];
      dist = fminf(dist, away[a] * r.perSafe[a]);
    }
    float steps = dist * r.perStep;
    if (!(fabsf(steps - rintf(steps)) > 1e-3f)) {
      dist = 1e30f;
#pragma unroll
      for (int a = 0; a < 3; a++) dist = fminf(dist, away[a] / safeAxis(r.rd[a]));
      steps = dist / r.stepSize;
    }
    s.next = fminf(t + fmaxf(1.f, floorf(steps) + 1.f) * r.stepSize, exit);
  }
  return s;
}
// The radiance a sample ds long adds per unit of the transmittance before it, and the factor it
// leaves of that transmittance.
template <class Cursor>
FP_DEV float4 shade(const SimParams& P, const FpRender& R, Cursor& c, const Ray& r, const Tint& tint, const Sample& s,
                    float ds) {
  const float texels = 1.f / (float)(P.B >> R.lightShift);  // lighting texels a cell: a power of two, exact
  float4 f = reconstruct(P, R, c, s.cell[0], s.cell[1], s.cell[2], s.filter);
  if (P.smokeDiv > 1) {  // fireProRenderField: the smoothed coarse density, trilinear
    const float q = 1.f / (float)P.smokeDiv;
    f.x = renderSmokeAt(P, R, c, s.cell[0] * q, s.cell[1] * q, s.cell[2] * q);
  }
  if (!(f.x + glowOf(f.z) > .002f)) return make_float4(0.f, 0.f, 0.f, 1.f);
  // fireProShade
  float3 glow = emissionOf(R, tint, f);
  float density = fmaxf(0.f, f.x) * R.optical[0];
  float sc[3] = {0.f, 0.f, 0.f};
  if (density > 0.f) {
    float4 inc = lightSample(P, R, c, s.cell[0] * texels, s.cell[1] * texels, s.cell[2] * texels);
    sc[0] = R.smoke[0] * (R.ambient[0] + R.sceneLight[0] * r.direct * inc.w + inc.x * .65f) * density;
    sc[1] = R.smoke[1] * (R.ambient[1] + R.sceneLight[1] * r.direct * inc.w + inc.y * .65f) * density;
    sc[2] = R.smoke[2] * (R.ambient[2] + R.sceneLight[2] * r.direct * inc.w + inc.z * .65f) * density;
  }
  float ext = extinctionOf(R, f);
  float tau = ext * ds;
  float integral = ds * (1.f - .5f * tau + tau * tau / 6.f);
  if (tau >= .001f) integral = (1.f - expf(-tau)) / ext;
  return make_float4((sc[0] + glow.x) * integral, (sc[1] + glow.y) * integral, (sc[2] + glow.z) * integral,
                     1.f - fminf(1.f, ext * integral));
}

// A ray is marched by a group of G lanes of a warp, a lane a step: the next G steps of the ray's
// lattice are looked up together, those before the first empty block (or the limit) are shaded
// together, and their colours and transmittances are composed over the lanes. A serial march is a
// chain of dependent lookups and loads a few hundred instructions long a step, and an image of a
// few tens of thousands of rays leaves the chip idle waiting for it; along the ray the lanes also
// read neighbouring cells and mostly agree on the filter. All lanes of a group hold the same ray
// state. The samples that count are the serial march's, at the very same positions; those past the
// point where the ray turns opaque are dropped.
// Every lane of the warp calls the two halves together, those without work with `on` false.
constexpr float OPAQUE = .008f;
struct March {
  float t, exit, trans, rad[3];
};
template <int G>
struct Steps {
  float t, ds;   // this lane's step
  float next;    // where the ray goes on after the group's steps
  bool lit, any; // this lane's block may hold something; some lane's of the group
  Sample s;
};
// The group's next steps before `limit`, looked up.
template <int G, class Cursor>
FP_DEV Steps<G> lookAhead(const SimParams& P, const FpRender& R, Cursor& c, const Ray& r, float limit, bool on,
                          const March& m) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & (G - 1);
  Steps<G> a;
  a.t = m.t;
#pragma unroll
  for (int j = 0; j < G - 1; j++)  // the serial march's own sums
    if (j < lane) a.t += r.stepSize;
  a.ds = fminf(r.stepSize, limit - a.t);
  const bool live = on && a.t < limit;
  a.s.lit = false;
  a.s.next = a.t;
  if (live) a.s = sampleAt(P, R, c, r, a.t, a.ds, m.exit);
  a.lit = live && a.s.lit;
  // Where the ray goes on: past the last step to shade, or past the empty block of the step after it.
  a.next = a.lit ? a.t + a.ds : a.s.next;
  a.any = a.lit;
  if constexpr (G > 1) {
    const int shift = (threadIdx.x & 31) & ~(G - 1);
    const unsigned lanes = (__ballot_sync(full, live) >> shift) & ((1u << G) - 1u);
    const unsigned dark = (~__ballot_sync(full, a.lit) >> shift) & ((1u << G) - 1u);
    const int n = dark ? __ffs((int)dark) - 1 : G;  // the steps to shade
    a.lit = a.lit && lane < n;
    a.any = n > 0;
    a.next = __shfl_sync(full, a.next, (n < G && ((lanes >> n) & 1u)) ? n : max(0, n - 1), G);
  }
  return a;
}
// The group's lit steps shaded and composed into the ray.
template <int G, class Cursor>
FP_DEV void shadeSteps(const SimParams& P, const FpRender& R, Cursor& c, const Ray& r, const Tint& tint, bool on,
                       const Steps<G>& a, March& m) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & (G - 1);
  float4 q = make_float4(0.f, 0.f, 0.f, 1.f);
  if (on && a.lit) q = shade(P, R, c, r, tint, a.s, a.ds);
  if constexpr (G > 1) {
    // The transmittance before each lane's step: an exclusive product over the group.
    float incl = q.w;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const float v = __shfl_up_sync(full, incl, o, G);
      if (lane >= o) incl *= v;
    }
    const float before = __shfl_up_sync(full, incl, 1, G);
    const float tb = lane == 0 ? m.trans : m.trans * before;
    // The steps before the first at which the serial march would have stopped count. (The transmittance
    // need not fall along the group: an opacity below zero raises it.)
    const unsigned stops = (__ballot_sync(full, !(tb >= OPAQUE)) >> ((threadIdx.x & 31) & ~(G - 1))) & ((1u << G) - 1u);
    const int n = stops ? __ffs((int)stops) - 1 : G;
    const bool counts = lane < n;
    float x = counts ? tb * q.x : 0.f, y = counts ? tb * q.y : 0.f, z = counts ? tb * q.z : 0.f;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      x += __shfl_xor_sync(full, x, o, G);
      y += __shfl_xor_sync(full, y, o, G);
      z += __shfl_xor_sync(full, z, o, G);
    }
    const float left = __shfl_sync(full, tb * q.w, max(0, n - 1), G);
    if (on) {
      m.rad[0] += x;
      m.rad[1] += y;
      m.rad[2] += z;
      m.trans = left;
    }
  } else if (on) {
    m.rad[0] += m.trans * q.x;
    m.rad[1] += m.trans * q.y;
    m.rad[2] += m.trans * q.z;
    m.trans *= q.w;
  }
}
// The march of the warp's rays, each from m.t to `end`: `limitOf()` gives the depth at which a
// ray's lattice starts over before the exit, `arrived()` is called whenever a ray has moved on.
// The rays of a warp cross their empty stretches together, by lookups alone, before any shades: a
// ray in empty space then does not wait, step by step, for the others' shading.
// What bounds it is instruction issue (cells come from L1): about 98 % L1 hits, DRAM idle. Slice
// pass, us: 14,400 rays of a small plume 2103 -> 82; 129,600 rays of a 1.8k-brick jet 8954 -> 801;
// 518,400 rays of 3.7k bricks 20,889 -> 2689; full resolution, 231,401 rays, quadratic 12,807 -> 722.
template <class Cursor, int G, class Limit, class Arrived>
FP_DEV void marchRays(const SimParams& P, const FpRender& R, const Ray& r, bool alive, float end, March& m, Limit limitOf,
                      Arrived arrived) {
  const unsigned full = 0xffffffffu;
  const Tint tint = tintOf(R);
  Cursor c = noBox<Cursor>();
  while (true) {
    Steps<G> a;
    bool ready = false;  // this group's steps hold a lit one
    a.next = 0.f;
    while (true) {
      alive = alive && m.t < end && m.trans >= OPAQUE;
      bool on = alive && !ready;
      if (on && m.t >= m.exit) {
        alive = enterBox(P, R, r, m.t, m.exit, c);
        on = alive && m.t < m.exit;
        if (alive) arrived();
      }
      if (!__any_sync(full, on)) {
        if (!__any_sync(full, alive && !ready)) break;
        continue;
      }
      Steps<G> b = lookAhead<G>(P, R, c, r, fminf(limitOf(), m.exit), on, m);
      if (on) {
        a = b;
        ready = b.any;
        if (!ready) {
          m.t = b.next;
          arrived();
        }
      }
    }
    if (!__any_sync(full, ready)) break;
    shadeSteps<G>(P, R, c, r, tint, ready, a, m);
    if (ready) {
      m.t = a.next;
      arrived();
    }
  }
}

// The pixel of a thread's group. A warp's rays and a CTA's four warps cover square tiles of the
// image, so that they read neighbouring bricks.
template <int G>
struct RayTile {
  static constexpr int RAYS = 32 / G;  // a warp's
  static constexpr int WX = RAYS >= 32 ? 8 : (RAYS >= 8 ? 4 : (RAYS >= 2 ? 2 : 1)), WY = RAYS / WX;
  static constexpr int TX = 2 * WX, TY = 2 * WY;
  static_assert(RTHREADS == 128, "four warps a CTA");
};
template <int G>
FP_DEV void groupPixel(int& px, int& py) {
  using T = RayTile<G>;
  const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) / G;
  px = blockIdx.x * T::TX + (warp & 1) * T::WX + g % T::WX;
  py = blockIdx.y * T::TY + (warp >> 1) * T::WY + g / T::WX;
}
template <int G>
static dim3 groupGrid(int w, int h) {
  using T = RayTile<G>;
  return dim3((unsigned)((w + T::TX - 1) / T::TX), (unsigned)((h + T::TY - 1) / T::TY));
}

// buildSlices (volume-slices.wgsl:28-122): a ray per half-resolution pixel marches from the
// first box entry to the last exit, box by box, recording radiance and opacity at FP_SLICES
// evenly spaced depths; depths passed by a skip or a jump between boxes keep the values of the
// moment, those past the exit or an opaque ray the final ones. Without a scene depth every pixel
// resumes from the last slice, so only that one is stored.
template <class Cursor, int G>
__global__ void __launch_bounds__(RTHREADS, MARCH_CTAS) k_slices(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  int px, py;
  groupPixel<G>(px, py);
  const bool inside = px < R.sliceW && py < R.sliceH;
  const size_t plane = (size_t)R.sliceW * R.sliceH;
  float4* out = R.slices + (size_t)py * R.sliceW + px;
  const bool writes = inside && (threadIdx.x & (G - 1)) == 0;
  March m{0.f, 0.f, 1.f, {0.f, 0.f, 0.f}};
  int recorded = 0;
  auto record = [&]() {
    if (writes && (R.depth || recorded == FP_SLICES - 1))
      out[(size_t)recorded * plane] = make_float4(m.rad[0], m.rad[1], m.rad[2], 1.f - m.trans);
    recorded++;
  };
  Ray r;
  bool alive = inside && R.boxCount > 0 &&
               rayOf(P, R, ((float)px + .5f) / (float)R.sliceW, ((float)py + .5f) / (float)R.sliceH, r);
  float spacing = 0.f, depth = 0.f;
  if (alive) {
    r.jitter = jitterOf((uint32_t)px, (uint32_t)py, R.time);
    spacing = fmaxf(r.hi - r.lo, 0.f) / (float)FP_SLICES;
    m.t = m.exit = r.lo;
    depth = r.lo + spacing;
  }
  marchRays<Cursor, G>(P, R, r, alive, r.hi, m, [&]() { return depth; },
               [&]() {
                 while (recorded < FP_SLICES && m.t >= depth) {
                   record();
                   depth = r.lo + spacing * (float)(recorded + 1);
                 }
               });
  while (recorded < FP_SLICES) record();
}

// fireProSceneVolume (scene-volume.wgsl:39-44, 146-167): the march of each pixel's ray up to
// the scene's depth through the boxes, from the last half-resolution slice in front of it when
// slices exist.
template <class Cursor, int G>
__global__ void __launch_bounds__(RTHREADS, MARCH_CTAS) k_march(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R) {
  const SimParams& P = *Pp;
  int px, py;
  groupPixel<G>(px, py);
  const bool inside = px < R.width && py < R.height;
  const size_t pix = (size_t)py * R.width + px;
  const float ux = ((float)px + .5f) / (float)R.width, uy = ((float)py + .5f) / (float)R.height;
  March m{0.f, 0.f, 1.f, {0.f, 0.f, 0.f}};
  Ray r;
  bool alive = inside && R.boxCount > 0 && rayOf(P, R, ux, uy, r);
  // fireProSceneDistance (volume-march.wgsl:76-89): the scene's depth ends the ray.
  float end = alive ? r.hi : 0.f;
  if (alive && R.depth) {
    const float d = R.depth[pix];
    if (d < .999999f) {
      const float cx = ux * 2.f - 1.f, cy = 1.f - uy * 2.f;
      const float* M = R.ivp;
      float hit[4];
      for (int k = 0; k < 4; k++) hit[k] = M[k] * cx + M[4 + k] * cy + M[8 + k] * d + M[12 + k];
      float dist = 0.f;
      for (int a = 0; a < 3; a++) dist += (hit[a] / hit[3] - r.ro[a]) * r.rd[a];
      end = fminf(end, dist);
    }
  }
  alive = alive && end > r.lo;
  if (alive) {
    r.jitter = jitterOf((uint32_t)px, (uint32_t)py, R.time);
    m.t = r.lo;
    if (R.slices) {
      // Resume from the last slice in front of the scene: the half-resolution texels
      // interpolated bilinearly (clamped at the edges) on that slice.
      const float count = (float)FP_SLICES;
      const float slice = R.depth ? floorf((end - r.lo) / (r.hi - r.lo) * count) : count;
      if (slice >= 1.f) {
        const int layer = (int)fminf(slice, count) - 1;
        float gx = ux * (float)R.sliceW - .5f, gy = uy * (float)R.sliceH - .5f;
        float fx0 = floorf(gx), fy0 = floorf(gy);
        float wx = gx - fx0, wy = gy - fy0;
        int x0 = (int)fx0, y0 = (int)fy0;
        int xs[2] = {min(max(x0, 0), R.sliceW - 1), min(max(x0 + 1, 0), R.sliceW - 1)};
        int ys[2] = {min(max(y0, 0), R.sliceH - 1), min(max(y0 + 1, 0), R.sliceH - 1)};
        const float4* S = R.slices + (size_t)layer * R.sliceW * R.sliceH;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < 4; k++) {
          int ix = k & 1, iy = k >> 1;
          add4(v, S[(size_t)ys[iy] * R.sliceW + xs[ix]], (ix ? wx : 1.f - wx) * (iy ? wy : 1.f - wy));
        }
        m.t = slice >= count ? r.hi : r.lo + (r.hi - r.lo) * slice / count;  // the last slice ends the ray
        m.trans = 1.f - v.w;
        m.rad[0] = v.x;
        m.rad[1] = v.y;
        m.rad[2] = v.z;
      }
    }
  }
  // fireProMarch: the cursor starts exited, so the first pass enters the box at t.
  const bool drawn = alive;
  m.exit = m.t;
  marchRays<Cursor, G>(P, R, r, alive, end, m, [&]() { return end; }, []() {});
  if (inside && (threadIdx.x & (G - 1)) == 0)
    reinterpret_cast<float4*>(R.image)[pix] =
        drawn ? make_float4(m.rad[0], m.rad[1], m.rad[2], 1.f - m.trans) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// collectLights (scene-lights.wgsl:37-106): a CTA of 64 lanes per computing brick, a lane per
// cell of the brick's 4^3 sample lattice (stride B/4, at the stride's middle). The brick's
// anchor is the nearest to its centre (height above an anchor counting a quarter; ties to the
// lower index); the lanes' luminance, luminance-weighted offsets and RGB are summed in shared
// memory and seven lanes add the totals to the anchor's floats.
__global__ void __launch_bounds__(64) k_collect_lights(const SimParams* __restrict__ Pp, const __grid_constant__ FpRender R,
                                                       const float* __restrict__ anchors, int count, float* sums) {
  const SimParams& P = *Pp;
  __shared__ float2 nearest[64];
  __shared__ float4 positions[64];
  __shared__ float4 colors[64];
  const uint32_t total = P.counters->active;
  const int lane = threadIdx.x, stride = P.B >> 2;
  const bool half = P.scalarHalf != 0;
  const float side = (float)P.B * P.h;
  const Tint tint = tintOf(R);
  for (uint32_t i = blockIdx.x; i < total; i += gridDim.x) {
    const uint32_t id = P.active[i];
    if (!homeOk(P, id)) continue;  // the bounds-checked build only
    const int e = P.entries[id];
    if (e < 0) continue;  // the same for the whole CTA
    const int slot = entryPage(e);
    const int4 t = __ldg(&P.tileRec[id >> 6]);
    const int l = id & 63;
    const int b[3] = {t.x * 4 + (l & 3), t.y * 4 + ((l >> 2) & 3), t.z * 4 + (l >> 4)};
    const int lx = (lane & 3) * stride + stride / 2, ly = ((lane >> 2) & 3) * stride + stride / 2,
              lz = (lane >> 4) * stride + stride / 2;
    const size_t o = (size_t)slot * 4 * P.N + (size_t)((lz * P.B + ly) * P.B + lx);
    float4 f = make_float4(ldHalf(P.fld, o, half), ldHalf(P.fld, o + P.N, half), ldHalf(P.fld, o + 2 * P.N, half),
                           ldHalf(P.fld, o + 3 * P.N, half));
    if (P.smokeDiv > 1) {
      // The coarse density sampled trilinearly at the cell's centre on the smoke lattice
      // (scene-lights.wgsl:59-65): a tap past the brick reads the +1 neighbour (the slot's
      // apron), zero without a slot; taps before the brick read zero.
      const int sh = P.smokeShift, S = 1 << sh, m = S - 1;
      const float r = 1.f / (float)P.smokeDiv;
      const float q[3] = {((float)lx + .5f) * r - .5f, ((float)ly + .5f) * r - .5f, ((float)lz + .5f) * r - .5f};
      int c0[3];
      float fr[3];
      for (int a = 0; a < 3; a++) {
        float g = floorf(q[a]);
        c0[a] = (int)g;
        fr[a] = q[a] - g;
      }
      float v = 0.f;
      for (int k = 0; k < 8; k++) {
        int d[3] = {k & 1, (k >> 1) & 1, k >> 2};
        int cl[3] = {c0[0] + d[0], c0[1] + d[1], c0[2] + d[2]};
        if (cl[0] < 0 || cl[1] < 0 || cl[2] < 0) continue;
        int nb[3] = {b[0] + (cl[0] >> sh), b[1] + (cl[1] >> sh), b[2] + (cl[2] >> sh)};
        int t = hashFind(P, nb[0] >> 2, nb[1] >> 2, nb[2] >> 2);
        int s = t < 0 ? -1 : checkSlot(P, FP_SITE_ENTRY, entryPage(P.entries[t * 64 + (((nb[2] & 3) * 4 + (nb[1] & 3)) * 4 + (nb[0] & 3))]));
        if (s < 0) continue;
        float w = (d[0] ? fr[0] : 1.f - fr[0]) * (d[1] ? fr[1] : 1.f - fr[1]) * (d[2] ? fr[2] : 1.f - fr[2]);
        v += ldHalf(P.smk, (size_t)s * P.smokeCells + ((((cl[2] & m) << sh) | (cl[1] & m)) << sh | (cl[0] & m)), half) * w;
      }
      f.x = v;
    }
    const float3 rgb = emissionOf(R, tint, f);
    const float luminance = rgb.x * .2126f + rgb.y * .7152f + rgb.z * .0722f;
    const float cx = ((float)b[0] + .5f) * side, cy = ((float)b[1] + .5f) * side, cz = ((float)b[2] + .5f) * side;
    float2 best = make_float2(1e38f, 0.f);
    for (int k = lane; k < count; k += 64) {
      float dx = cx - anchors[3 * k], dy = cy - anchors[3 * k + 1], dz = cz - anchors[3 * k + 2];
      float rise = dy > 0.f ? dy * .25f : dy;
      float d = dx * dx + dz * dz + rise * rise;
      if (d < best.x) best = make_float2(d, (float)k);
    }
    nearest[lane] = best;
    __syncthreads();
    for (int reach = 32; reach > 0; reach >>= 1) {
      if (lane < reach) {
        float2 other = nearest[lane + reach], mine = nearest[lane];
        if (other.x < mine.x || (other.x == mine.x && other.y < mine.y)) nearest[lane] = other;
      }
      __syncthreads();
    }
    const int anchor = (int)nearest[0].y;
    const float px = ((float)(b[0] * P.B + lx) + .5f) * P.h, py = ((float)(b[1] * P.B + ly) + .5f) * P.h,
                pz = ((float)(b[2] * P.B + lz) + .5f) * P.h;
    positions[lane] = make_float4(luminance, (px - anchors[3 * anchor]) * luminance,
                                  (py - anchors[3 * anchor + 1]) * luminance, (pz - anchors[3 * anchor + 2]) * luminance);
    colors[lane] = make_float4(rgb.x, rgb.y, rgb.z, 0.f);
    __syncthreads();
    for (int reach = 32; reach > 0; reach >>= 1) {
      if (lane < reach) {
        float4 a = positions[lane], c = positions[lane + reach], u = colors[lane], v = colors[lane + reach];
        positions[lane] = make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w + c.w);
        colors[lane] = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, 0.f);
      }
      __syncthreads();
    }
    if (lane < 7) {
      const float totals[7] = {positions[0].x, positions[0].y, positions[0].z, positions[0].w,
                               colors[0].x, colors[0].y, colors[0].z};
      atomicAdd(&sums[anchor * 8 + lane], totals[lane]);
    }
    __syncthreads();  // the shared sums are read before the next brick's lanes write them
  }
}

}  // namespace

void fp_launch_collect_lights(const SimParams* dP, const FpRender& R, const float* anchors, int count, float* sums,
                              int sms, cudaStream_t st) {
  k_collect_lights<<<sms * 16, 64, 0, st>>>(dP, R, anchors, count, sums);
}

// Lanes a ray (marchRays): enough that the rays' lanes fill the chip several times over (148 SMs x
// 12 warps), no more, since a group's lanes share the ray's own work and its last steps leave lanes
// idle. What is best moves with the scene and with the steps a ray takes; the lines lie where the means
// over five scenes, both resolutions and 128 and 256 steps cross. A render relative to its best number
// of lanes, the mean at half resolution, 128 / 256 steps:
//   rays          1           2           4           8           16
//   9,216     2.39/3.08   1.60/1.89   1.19/1.35   1.01/1.06   1.01/1.01
//   17,280    2.12/2.59   1.43/1.59   1.09/1.17   1.00/1.00   1.07/1.04
//   30,720    1.71/2.14   1.17/1.32   1.01/1.02   1.05/1.01   1.18/1.12
//   43,200    1.63/1.95   1.12/1.30   1.00/1.00   1.08/1.04   1.27/1.20
//   86,400    1.24/1.43   1.02/1.05   1.05/1.02   1.23/1.15   1.58/1.43
//   129,600   1.09/1.22   1.00/1.01   1.10/1.07   1.35/1.27   1.81/1.65
//   230,400   1.02/1.03   1.06/1.04   1.24/1.17   1.61/1.46   2.26/1.95
//   518,400   1.02/1.02   1.11/1.08   1.38/1.27   1.88/1.67   2.77/2.34
// Past 230,400 one lane would be better in most scenes and worse in the largest (518,400 rays of 256 steps
// through 3.7k bricks: 3962 us, with two 3829); from 921,600 on in nearly all, by a tenth.
template <class Cursor, int G>
static void marchLaunch(const SimParams* dP, const FpRender& R, cudaStream_t st) {
  if (R.slices) {
    k_slices<Cursor, G><<<groupGrid<G>(R.sliceW, R.sliceH), RTHREADS, 0, st>>>(dP, R);
    // Every pixel resumes at its last slice: at most an eighth of its ray is left to march.
    k_march<Cursor, 1><<<groupGrid<1>(R.width, R.height), RTHREADS, 0, st>>>(dP, R);
  } else {
    k_march<Cursor, G><<<groupGrid<G>(R.width, R.height), RTHREADS, 0, st>>>(dP, R);
  }
}
template <class Cursor>
static void poolsLaunch(const SimParams* dP, const FpRender& R, int sms, cudaStream_t st) {
  k_render_field<Cursor><<<sms * 24, RTHREADS, 0, st>>>(dP, R);
  // More CTAs than reside: texels that nothing is at cost little, so equal shares of them are not
  // equal work (on the default grid 5 CTAs an SM took 16 % longer than 40, 20 took 2 %).
  k_render_light<Cursor><<<sms * 40, RTHREADS, 0, st>>>(dP, R);
  if (R.units)
    k_render_occupancy<Cursor, true><<<sms * 8, RTHREADS, 0, st>>>(dP, R);
  else
    k_render_occupancy<Cursor, false><<<sms * 8, RTHREADS, 0, st>>>(dP, R);
}
void fp_launch_render(const SimParams* dP, const FpRender& R, int sms, cudaStream_t st) {
  if (!R.pages) {
    // Rare, so one form for every size: 2 and 4 lanes a ray 2220 and 1803 us (14,400 rays), 6.3 and 4.5 ms
    // (129,600), 8.9 and 6.5 (231,401), 21.3 and 22.8 (518,400).
    poolsLaunch<HashCursor>(dP, R, sms, st);
    marchLaunch<HashCursor, 4>(dP, R, st);
    return;
  }
  const int rows = R.boxCount < 64 ? R.boxCount : 64;
  const long long blocks = (R.pageCount / rows + 255) / 256;
  const dim3 grid((unsigned)(blocks < 1 ? 1 : (blocks < sms * 8 ? blocks : sms * 8)), rows);
  k_render_pages<<<grid, 256, 0, st>>>(dP, R);
  if (R.apronCap) k_render_aprons<<<grid, 256, 0, st>>>(R);
  poolsLaunch<TableCursor>(dP, R, sms, st);
  const long long rays = R.slices ? (long long)R.sliceW * R.sliceH : (long long)R.width * R.height;
  if (rays >= 100000)
    marchLaunch<TableCursor, 2>(dP, R, st);
  else if (rays >= 36000)
    marchLaunch<TableCursor, 4>(dP, R, st);
  else if (rays >= 16000)
    marchLaunch<TableCursor, 8>(dP, R, st);
  else
    marchLaunch<TableCursor, 16>(dP, R, st);
}
