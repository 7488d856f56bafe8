// Sparse geometric multigrid for the pressure (src/engine/shaders/pressure.wgsl and
// src/engine/PressureSolver.ts). Level 0 is the velocity grid; each brick holds levels down
// to 2^3 cells; three tile levels (4^3, 2^3 and one cell per tile) follow. Weighted Jacobi
// (omega 0.8) smoothing, residual restriction that also writes the coarse level's first
// iterate, trilinear prolongation with Neumann ghosts at solid coarse cells, and a bottom
// solve in one CTA. Brick levels run a CTA per computing brick; tile levels a CTA per tile.
#include "fp_device.cuh"
#include "fp_launch.h"
#include "fp_overlap.cuh"

namespace {

constexpr uint32_t SOLIDF = 1024u;

FP_DEV int levelShift(const SimParams& P, int level) {
  return level < P.brickLevels ? P.brickLevels - level : P.brickLevels + 2 - level;
}

// cellAddress (pressure.wgsl:72-92): -1 without storage.
FP_DEV long cellAddress(const SimParams& P, const Home& H, int px, int py, int pz, int level) {
  int s = levelShift(P, level), side = 1 << s, m = side - 1;
  long owner;
  if (level < P.brickLevels) {
    int slot = brickSlot(P, H, px >> s, py >> s, pz >> s);
    if (slot < 0) return -1;
    owner = slot;
  } else {
    // Multigrid homes are live tiles, and a live tile is its own centre neighbour.
    int tx = px >> s, ty = py >> s, tz = pz >> s;
    int t = (tx == H.tx && ty == H.ty && tz == H.tz && H.tile >= 0) ? H.tile : tileAt(P, H, tx, ty, tz);
    if (t < 0) return -1;
    owner = t;
  }
  return owner * side * side * side + ((pz & m) * side + (py & m)) * side + (px & m);
}

// Whether cell (px,py,pz) of tile level `level` is a pressure unknown: every brick it covers
// computes, from the tile's mask of computing bricks (k_tile_masks, this step).
FP_DEV bool tileCellActive(const SimParams& P, const Home& H, int px, int py, int pz, int level) {
  int s = levelShift(P, level), side = 1 << s;
  int tx = px >> s, ty = py >> s, tz = pz >> s;
  int t = (tx == H.tx && ty == H.ty && tz == H.tz && H.tile >= 0) ? H.tile : tileAt(P, H, tx, ty, tz);
  if (t < 0) return false;
  uint64_t m = P.tileMask[t];
  int lx = px & (side - 1), ly = py & (side - 1), lz = pz & (side - 1);
  if (side == 4) return (m >> ((lz * 4 + ly) * 4 + lx)) & 1ull;  // a cell per brick
  if (side == 2) {                                                   // 2^3 bricks a cell
    uint64_t c = 0x0000000000330033ull << (2 * lx + 8 * ly + 32 * lz);
    return (m & c) == c;
  }
  return m == ~0ull;  // the whole tile
}

// activeCell (pressure.wgsl:100-136): whether a level's cell is a pressure unknown.
FP_DEV bool activeCell(const SimParams& P, const Home& H, int px, int py, int pz, int level) {
  int bl = P.brickLevels;
  if (level >= bl) return tileCellActive(P, H, px, py, pz, level);  // every covered brick computes
  int span = 1 << level;
  int lx = (px * span - 1) >> bl, ly = (py * span - 1) >> bl, lz = (pz * span - 1) >> bl;
  int hx = (px * span + span - 1) >> bl, hy = (py * span + span - 1) >> bl, hz = (pz * span + span - 1) >> bl;
  if (P.ground) ly = max(ly, 0);
  for (int z = lz; z <= hz; z++)
    for (int y = ly; y <= hy; y++)
      for (int x = lx; x <= hx; x++)
        if (brickSlot(P, H, x, y, z) < 0) return false;
  return true;
}

FP_DEV uint32_t expandFlags(uint8_t t) { return (t & FP_STORED_SOLID) ? SOLIDF : (uint32_t)(t & 63u); }
FP_DEV float diagOf(uint32_t f) {
  return (float)((f >> 0) & 1u) + (float)((f >> 1) & 1u) + ((float)((f >> 2) & 1u) + (float)((f >> 3) & 1u)) +
         ((float)((f >> 4) & 1u) + (float)((f >> 5) & 1u));
}
// Levels above the finest hold BF16 values in FP_PRECISION_MIXED.
FP_DEV bool narrowLevel(const SimParams& P, int level) { return level > 0 && P.coarseBf16 != 0; }
FP_DEV float readAt(const SimParams& P, const Home& H, const float* arr, int px, int py, int pz, int level) {
  if (!arr) return 0.f;  // a relaxation from zero
  long a = cellAddress(P, H, px, py, pz, level);
  return a < 0 ? 0.f : ldBf(arr, a, narrowLevel(P, level));
}
// stencil (pressure.wgsl:360-402): open neighbours' sum; cubic cells weigh 1 on every axis.
FP_DEV float stencilSum(const SimParams& P, const Home& H, const float* p, int px, int py, int pz, uint32_t f,
                        int level) {
  float v0 = (f & 1u) ? readAt(P, H, p, px + 1, py, pz, level) : 0.f;
  float v1 = (f & 2u) ? readAt(P, H, p, px - 1, py, pz, level) : 0.f;
  float v2 = (f & 4u) ? readAt(P, H, p, px, py + 1, pz, level) : 0.f;
  float v3 = (f & 8u) ? readAt(P, H, p, px, py - 1, pz, level) : 0.f;
  float v4 = (f & 16u) ? readAt(P, H, p, px, py, pz + 1, level) : 0.f;
  float v5 = (f & 32u) ? readAt(P, H, p, px, py, pz - 1, level) : 0.f;
  return (v0 + v1) + (v2 + v3) + (v4 + v5);
}

FP_DEV bool coarseSolid(const SimParams& P, const Home& H, int px, int py, int pz, int level) {
  long a = cellAddress(P, H, px, py, pz, level);
  if (a < 0) return false;
  return (P.topo[level][a] & FP_STORED_SOLID) != 0;
}
// coarseValue (pressure.wgsl:670-696): Neumann ghosts at solid coarse cells, the ground mirrored.
FP_DEV float coarseValue(const SimParams& P, const Home& H, const float* coarse, int level, int px, int py, int pz) {
  int groundY = P.ground ? 0 : -0x7fffffff;
  int c[3] = {px, max(py, groundY), pz};
  if (!coarseSolid(P, H, c[0], c[1], c[2], level)) return readAt(P, H, coarse, c[0], c[1], c[2], level);
  float sum = 0.f, count = 0.f;
  for (int axis = 0; axis < 3; axis++)
    for (int side = -1; side <= 1; side += 2) {
      int q[3] = {c[0], c[1], c[2]};
      q[axis] += side;
      q[1] = max(q[1], groundY);
      if (!coarseSolid(P, H, q[0], q[1], q[2], level)) {
        sum += readAt(P, H, coarse, q[0], q[1], q[2], level);
        count += 1.f;
      }
    }
  return sum / fmaxf(count, 1.f);
}

// Operation on one cell of a level (relaxCell, prolongateCell, restrictCell).
enum Op { RELAX = 0, PROLONG = 1, RESTRICT = 2 };

struct Args {
  int level;  // output level
  const float* rhs;
  const float* pin;
  const float* coarse;
  float* pout;
  float* cfirst;
  bool rhsN, pinN, coarseN, poutN, cfirstN;  // the buffer holds BF16
  bool skip;                                 // a later V-cycle of a converged solve: no work
  int colour, halves;                        // MgSel::colour, MgSel::halves
};

// A launch names its buffers by selector, level * 4 + which (0 and 1 the level's pressure
// pair, 2 its right-hand side; -1 none), and each simulation of the batch resolves them.
FP_DEV float* mgBuffer(const SimParams& P, int sel) {
  if (sel < 0) return nullptr;
  int level = sel >> 2, which = sel & 3;
  if (which == 2) return level == 0 ? P.div : P.lrhs[level];
  if (which == 3) return level == 0 ? P.kry[0] : nullptr;
  return level == 0 ? P.p0[which] : P.lp[level][which];
}
FP_DEV Args resolve(const SimParams& P, const MgSel& S) {
  Args A;
  A.level = S.level;
  A.rhs = mgBuffer(P, S.rhs);
  A.pin = mgBuffer(P, S.pin);
  A.coarse = mgBuffer(P, S.coarse);
  A.pout = mgBuffer(P, S.pout);
  A.cfirst = mgBuffer(P, S.cfirst);
  A.rhsN = S.rhs >= 0 && narrowLevel(P, S.rhs >> 2);
  A.pinN = S.pin >= 0 && narrowLevel(P, S.pin >> 2);
  A.coarseN = S.coarse >= 0 && narrowLevel(P, S.coarse >> 2);
  A.poutN = S.pout >= 0 && narrowLevel(P, S.pout >> 2);
  A.cfirstN = S.cfirst >= 0 && narrowLevel(P, S.cfirst >> 2);
  A.skip = S.cycle > 0 && P.solver->converged != 0;
  A.colour = S.colour;
  A.halves = S.halves;
  return A;
}

// Red-black: the cell's colour, 0 for x + y + z even.
FP_DEV int parityOf(int px, int py, int pz) { return (px + py + pz) & 1; }

FP_DEV void relaxCell(const SimParams& P, const Home& H, const Args& A, long a, int px, int py, int pz) {
  if (A.colour != 0 && parityOf(px, py, pz) != A.colour - 1) {
    // Red-black, the other colour: kept, or zero when the level starts from zero.
    if (!A.pin) stBf(A.pout, a, 0.f, A.poutN);
    return;
  }
  uint32_t f = expandFlags(P.topo[A.level][a]);
  if ((f & SOLIDF) || !activeCell(P, H, px, py, pz, A.level)) {
    stBf(A.pout, a, 0.f, A.poutN);
    return;
  }
  float sum = A.pin ? stencilSum(P, H, A.pin, px, py, pz, f, A.level) : 0.f;
  float cand = (sum - ldBf(A.rhs, a, A.rhsN)) / fmaxf(diagOf(f), 1e-12f);
  if (A.colour != 0)
    stBf(A.pout, a, cand, A.poutN);  // Gauss-Seidel in place
  else
    stBf(A.pout, a, mixf(A.pin ? ldBf(A.pin, a, A.pinN) : 0.f, cand, 0.8f), A.poutN);
}

FP_DEV void prolongCell(const SimParams& P, const Home& H, const Args& A, long a, int px, int py, int pz) {
  uint32_t f = expandFlags(P.topo[A.level][a]);
  if ((f & SOLIDF) || !activeCell(P, H, px, py, pz, A.level)) {
    stBf(A.pout, a, 0.f, A.poutN);
    return;
  }
  int cl = A.level + 1;
  float qx = ((float)px + 0.5f) * 0.5f - 0.5f, qy = ((float)py + 0.5f) * 0.5f - 0.5f, qz = ((float)pz + 0.5f) * 0.5f - 0.5f;
  int ix = (int)floorf(qx), iy = (int)floorf(qy), iz = (int)floorf(qz);
  float fx = qx - floorf(qx), fy = qy - floorf(qy), fz = qz - floorf(qz);
  bool fast = P.colliderCount == 0 && (!P.ground || iy >= 0);
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
    v[k] = fast ? readAt(P, H, A.coarse, ix + dx, iy + dy, iz + dz, cl)
                : coarseValue(P, H, A.coarse, cl, ix + dx, iy + dy, iz + dz);
  }
  float corr = mixf(mixf(mixf(v[0], v[1], fx), mixf(v[2], v[3], fx), fy), mixf(mixf(v[4], v[5], fx), mixf(v[6], v[7], fx), fy),
                    fz);
  stBf(A.pout, a, ldBf(A.pin, a, A.pinN) + corr, A.poutN);
}

// restrictCell (pressure.wgsl:601-647): (cx,cy,cz) is a cell of the coarse (output) level.
FP_DEV void restrictCell(const SimParams& P, const Home& H, const Args& A, long out, int cx, int cy, int cz) {
  int fine = A.level - 1;
  float residual = 0.f;
  bool every = true;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int px = cx * 2 + (k & 1), py = cy * 2 + ((k >> 1) & 1), pz = cz * 2 + (k >> 2);
    bool unknown = activeCell(P, H, px, py, pz, fine);
    every = every && unknown;
    if (unknown) {
      long a = cellAddress(P, H, px, py, pz, fine);
      uint32_t f = expandFlags(P.topo[fine][a]);
      if (!(f & SOLIDF)) {
        float sum = stencilSum(P, H, A.pin, px, py, pz, f, fine);
        residual += ldBf(A.rhs, a, A.rhsN) - (sum - diagOf(f) * ldBf(A.pin, a, A.pinN));
      }
    }
  }
  float r = residual * 0.5f;
  stBf(A.pout, out, r, A.poutN);  // the coarse right-hand side
  float first = 0.f;
  if (every) {
    uint32_t f = expandFlags(P.topo[A.level][out]);
    if (!(f & SOLIDF)) first = mixf(0.f, (0.f - r) / fmaxf(diagOf(f), 1e-12f), 0.8f);
  }
  stBf(A.cfirst, out, first, A.cfirstN);
}

template <int OP>
FP_DEV void levelCell(const SimParams& P, const Home& H, const Args& A, long a, int px, int py, int pz) {
  if (OP == RELAX) relaxCell(P, H, A, a, px, py, pz);
  if (OP == PROLONG) prolongCell(P, H, A, a, px, py, pz);
  if (OP == RESTRICT) restrictCell(P, H, A, a, px, py, pz);
}

// Staged brick levels. A CTA copies, for its bricks, the values of the level it reads plus a
// rim into shared memory, and once per brick whether each negative-octant neighbour brick
// computes; the cell operations then read no directory. Same arithmetic, same order as
// relaxCell / restrictCell / prolongCell above.
//   RELAX     stage A.pin at A.level;           write A.pout at A.level
//   RESTRICT  stage A.pin at A.level - 1 (fine); write A.pout, A.cfirst at A.level (coarse)
//   PROLONG   stage A.coarse at A.level + 1;    write A.pout at A.level
// SB, the staged level's cells per brick side, fixes every shape at compile time; SB = 1 is
// the first tile level (one cell per brick), which prolongation stages through the tiles.
template <int OP, int SB>
struct Staged {
  static constexpr int R = OP == PROLONG ? 2 : 1;  // rim: prolongation's Neumann ghosts reach two
  static constexpr int S = SB + 2 * R, S2 = S * S, S3 = S2 * S;
  static constexpr int FS = OP == PROLONG ? 2 * SB : SB;  // the fine level's side
  static constexpr int OS = OP == RESTRICT ? SB / 2 : FS;  // the output level's side
  static constexpr int OUT = OS * OS * OS;
  static constexpr int GROUP = OUT >= 256 ? 256 : (OUT >= 64 ? 64 : 32);  // threads per brick
  static constexpr int NG = 256 / GROUP;                                  // bricks per CTA
  static constexpr int WORDS = S3 + (OP == PROLONG ? (S3 + 3) / 4 : 0);   // values + solid bytes
  static constexpr size_t SMEM = (size_t)NG * WORDS * sizeof(float);
};
constexpr int log2c(int v) { return v <= 1 ? 0 : 1 + log2c(v / 2); }

template <int OP, int SB>
__global__ void __launch_bounds__(256) k_level_bricks_staged(FpBatch bt, MgSel Sl) {
  using K = Staged<OP, SB>;
  constexpr int S = K::S, S2 = K::S2, S3 = K::S3, R = K::R, GROUP = K::GROUP, NG = K::NG;
  constexpr int FS = K::FS, fs = log2c(FS), FCELLS = FS * FS * FS;
  __shared__ int nslotAll[NG][27];
  __shared__ int needAll[NG][8];  // bit k of the index: -1 on axis k
  extern __shared__ float stAll[];
  const int g = threadIdx.x / GROUP, t = threadIdx.x % GROUP;
  int* nslot = nslotAll[g];
  int* need = needAll[g];
  float* st = stAll + g * K::WORDS;
  uint8_t* solidSt = reinterpret_cast<uint8_t*>(st + S3);
  uint32_t total = workTotal(bt, FP_WORK_ACTIVE);
  for (uint32_t base = blockIdx.x * NG; base < total; base += gridDim.x * NG) {
    uint32_t item = base + g;
    uint32_t i;
    const SimParams& P = *workSim(bt, FP_WORK_ACTIVE, item < total ? item : base, i).vview;
    const Args A = resolve(P, Sl);
    const bool has = item < total && !A.skip && homeOk(P, P.active[i]);  // homeOk: the bounds-checked build
    const int fineLevel = OP == RESTRICT ? A.level - 1 : A.level;
    const int stageLevel = OP == PROLONG ? A.level + 1 : fineLevel;
    const float* src = OP == PROLONG ? A.coarse : A.pin;
    const bool srcN = OP == PROLONG ? A.coarseN : A.pinN;
    const uint32_t id = has ? P.active[i] : 0u;
    Home H = homeOf(P, id, nslot);
    if (has && t < 27) nslot[t] = checkSlot(P, FP_SITE_RECORD, entryPage(P.records[(size_t)id * FP_RECORD_WORDS + t]));
    __syncthreads();
    const int ox = H.bx * SB - R, oy = H.by * SB - R, oz = H.bz * SB - R;
    // Relaxation and prolongation: this thread's own cells' flags and right-hand side or
    // current value, loaded before the stage so that both sets of loads are in flight together.
    constexpr int K = OP == RESTRICT ? 1 : (FCELLS + GROUP - 1) / GROUP;
    uint8_t ownTopo[K];
    float ownValue[K];
    if (OP != RESTRICT && has) {
      const long slot0 = nslot[13];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int o = t + k * GROUP;
        if (o < FCELLS) {
          const long a = slot0 * FCELLS + o;
          ownTopo[k] = P.topo[fineLevel][a];
          ownValue[k] = OP == RELAX ? ldBf(A.rhs, a, A.rhsN) : ldBf(A.pin, a, A.pinN);
        }
      }
    }
    bool solidStaged = false;  // prolongation: a solid coarse cell in this thread's stage cells
    if (has) {
      if (t < 8) {
        int dx = -(t & 1), dy = -((t >> 1) & 1), dz = -(t >> 2);
        bool below = P.ground && H.by + dy < 0;
        need[t] = below || nslot[nbrIndex(dx, dy, dz)] >= 0;
      }
      for (int q = t; q < S3; q += GROUP) {
        const int lx = q % S, ly = (q / S) % S, lz = q / S2;
        long a;
        if (SB > 1) {
          // Brick levels: the neighbour brick from the record, the cell within it.
          const int dx = lx < R ? -1 : (lx >= R + SB ? 1 : 0), dy = ly < R ? -1 : (ly >= R + SB ? 1 : 0),
                    dz = lz < R ? -1 : (lz >= R + SB ? 1 : 0);
          const int s = nslot[nbrIndex(dx, dy, dz)];
          const int cx = (lx - R) & (SB - 1), cy = (ly - R) & (SB - 1), cz = (lz - R) & (SB - 1);
          a = s < 0 ? -1 : (long)s * (SB * SB * SB) + (cz * SB + cy) * SB + cx;
        } else {
          a = cellAddress(P, H, ox + lx, oy + ly, oz + lz, stageLevel);
        }
        // A relaxation from zero stages nothing; a red-black half-sweep stages only the other
        // colour (a cell of the colour it writes reads none of its own colour).
        const bool skipLoad = OP == RELAX && (!src || (A.colour != 0 && ((ox + oy + oz + lx + ly + lz) & 1) == A.colour - 1));
        st[q] = (a < 0 || skipLoad) ? 0.f : ldBf(src, a, srcN);
        if (OP == PROLONG) {
          const bool solid = a >= 0 && (P.topo[stageLevel][a] & FP_STORED_SOLID);
          solidSt[q] = solid ? 1 : 0;
          solidStaged = solidStaged || solid;
        }
      }
    }
    // Without a solid coarse cell anywhere in the CTA's stages a Neumann ghost is the staged
    // value itself (coarseValue's first test), so prolongation may read the stage directly.
    bool anySolid = false;
    if (OP == PROLONG)
      anySolid = __syncthreads_or(solidStaged) != 0;
    else
      __syncthreads();
    if (has) {
      // The negative-octant neighbours that compute, as bits; a fine cell on the brick's low
      // faces is an unknown when every neighbour its faces touch computes (activeCell).
      uint32_t needBits = 0;
#pragma unroll
      for (int k = 0; k < 8; k++) needBits |= need[k] ? 1u << k : 0u;
      auto unknown = [&](int lx, int ly, int lz) {
        uint32_t sub = 1u;  // the octants k whose set axes are all on a low face here
        if (lx == 0) sub |= sub << 1;
        if (ly == 0) sub |= sub << 2;
        if (lz == 0) sub |= sub << 4;
        return (~needBits & sub) == 0u;
      };
      // coarseValue (pressure.wgsl:670-696) from the stage.
      auto ghost = [&](int cx, int cy, int cz) {
        int groundY = P.ground ? 0 : -0x7fffffff;
        int c[3] = {cx, max(cy, groundY), cz};
        auto at = [&](int x, int y, int z) { return ((z - oz) * S + (y - oy)) * S + (x - ox); };
        int ci = at(c[0], c[1], c[2]);
        if (!solidSt[ci]) return st[ci];
        float sum = 0.f, count = 0.f;
        for (int axis = 0; axis < 3; axis++)
          for (int side = -1; side <= 1; side += 2) {
            int q[3] = {c[0], c[1], c[2]};
            q[axis] += side;
            q[1] = max(q[1], groundY);
            int qi = at(q[0], q[1], q[2]);
            if (!solidSt[qi]) {
              sum += st[qi];
              count += 1.f;
            }
          }
        return sum / fmaxf(count, 1.f);
      };
      const long slot = nslot[13];
      // Stencil sum of the open sides of a fine cell, from the stage (RELAX, RESTRICT).
      auto sumAt = [&](int lx, int ly, int lz, uint32_t f) {
        int c = ((lz + 1) * S + (ly + 1)) * S + (lx + 1);
        float v0 = (f & 1u) ? st[c + 1] : 0.f, v1 = (f & 2u) ? st[c - 1] : 0.f;
        float v2 = (f & 4u) ? st[c + S] : 0.f, v3 = (f & 8u) ? st[c - S] : 0.f;
        float v4 = (f & 16u) ? st[c + S2] : 0.f, v5 = (f & 32u) ? st[c - S2] : 0.f;
        return (v0 + v1) + (v2 + v3) + (v4 + v5);
      };
      if (OP == RELAX || OP == PROLONG) {
#pragma unroll
        for (int k = 0; k < K; k++) {
          const int o = t + k * GROUP;
          if (o >= FCELLS) break;
          const int lx = o & (FS - 1), ly = (o >> fs) & (FS - 1), lz = o >> (2 * fs);
          const long a = slot * FCELLS + o;
          if (OP == RELAX && A.colour != 0 &&
              ((H.bx * FS + lx + H.by * FS + ly + H.bz * FS + lz) & 1) != A.colour - 1) {
            // Red-black, the other colour: kept, or zero when the level starts from zero.
            if (!src) stBf(A.pout, a, 0.f, A.poutN);
            continue;
          }
          uint32_t f = expandFlags(ownTopo[k]);
          if ((f & SOLIDF) || !unknown(lx, ly, lz)) {
            stBf(A.pout, a, 0.f, A.poutN);
            continue;
          }
          if (OP == RELAX) {
            float cand = (sumAt(lx, ly, lz, f) - ownValue[k]) / fmaxf(diagOf(f), 1e-12f);
            if (A.colour != 0) {
              stBf(A.pout, a, cand, A.poutN);  // Gauss-Seidel in place
            } else {
              float center = st[((lz + 1) * S + (ly + 1)) * S + (lx + 1)];
              stBf(A.pout, a, mixf(center, cand, 0.8f), A.poutN);
            }
          } else {
            int px = H.bx * FS + lx, py = H.by * FS + ly, pz = H.bz * FS + lz;
            float qx = ((float)px + 0.5f) * 0.5f - 0.5f, qy = ((float)py + 0.5f) * 0.5f - 0.5f,
                  qz = ((float)pz + 0.5f) * 0.5f - 0.5f;
            int ix = (int)floorf(qx), iy = (int)floorf(qy), iz = (int)floorf(qz);
            float fx = qx - floorf(qx), fy = qy - floorf(qy), fz = qz - floorf(qz);
            bool fast = (P.colliderCount == 0 || !anySolid) && (!P.ground || iy >= 0);
            // Below the ground the mirrored ghosts read the row above it, which a brick under
            // y = 0 does not stage: those read through the directory.
            bool staged = !(P.ground && H.by < 0);
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
              int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
              v[q] = fast     ? st[((iz + dz - oz) * S + (iy + dy - oy)) * S + (ix + dx - ox)]
                     : staged ? ghost(ix + dx, iy + dy, iz + dz)
                              : coarseValue(P, H, A.coarse, A.level + 1, ix + dx, iy + dy, iz + dz);
            }
            float corr = mixf(mixf(mixf(v[0], v[1], fx), mixf(v[2], v[3], fx), fy),
                              mixf(mixf(v[4], v[5], fx), mixf(v[6], v[7], fx), fy), fz);
            stBf(A.pout, a, ownValue[k] + corr, A.poutN);
          }
        }
      } else {  // RESTRICT: coarse cells of this brick at A.level
        constexpr int cside = FS / 2, cs = fs - 1, ccells = cside * cside * cside;
        for (int o = t; o < ccells; o += GROUP) {
          const int cx = o & (cside - 1), cy = (o >> cs) & (cside - 1), cz = o >> (2 * cs);
          float residual = 0.f;
          bool every = true;
#pragma unroll
          for (int k = 0; k < 8; k++) {
            int lx = cx * 2 + (k & 1), ly = cy * 2 + ((k >> 1) & 1), lz = cz * 2 + (k >> 2);
            bool u = unknown(lx, ly, lz);
            every = every && u;
            if (u) {
              long a = slot * FCELLS + (((lz << fs) | ly) << fs | lx);
              uint32_t f = expandFlags(P.topo[fineLevel][a]);
              if (!(f & SOLIDF)) {
                float center = st[((lz + 1) * S + (ly + 1)) * S + (lx + 1)];
                residual += ldBf(A.rhs, a, A.rhsN) - (sumAt(lx, ly, lz, f) - diagOf(f) * center);
              }
            }
          }
          float r = residual * 0.5f;
          // From the last brick level (2^3 a brick) the coarse level is the first tile level,
          // one cell a brick at the brick's own id (tile slot x 64 + its place in the tile).
          const long out = SB == 2 ? (long)id : slot * ccells + o;
          stBf(A.pout, out, r, A.poutN);
          float first = 0.f;
          if (every) {
            uint32_t f = expandFlags(P.topo[A.level][out]);
            if (!(f & SOLIDF)) first = mixf(0.f, (0.f - r) / fmaxf(diagOf(f), 1e-12f), 0.8f);
          }
          stBf(A.cfirst, out, first, A.cfirstN);
        }
      }
    }
    __syncthreads();
  }
}


FP_DEV Home enterTile(const SimParams& P, int t, int4 rec) {
  Home H;
  H.tile = t;
  H.tx = rec.x;
  H.ty = rec.y;
  H.tz = rec.z;
  H.bx = H.by = H.bz = -(1 << 29);  // no home brick: lookups go through the tiles
  H.nslot = nullptr;
  return H;
}

// The Jacobi V-cycle's work on a level in one launch a leg: a CTA stages a box of values three cells
// beyond what it owns, and works on it there, each sweep a cell less far out, until the last covers
// its own cells. The cells of the rim are worked on by their own CTA too, with the same arithmetic
// from the same values (each step's result rounded as the level stores it), so all agree. The result
// goes to the level's other buffer, since the neighbours read this one.
//   REST   the restriction alone (the finest level, whose first iterate the divergence left)
//   DOWN   two sweeps (written: prolongation adds to them) and the restriction of the result
//   UP     three sweeps
//   PUP    prolongation from the level below, and three sweeps
//   RB     red-black, a box four cells out: one or two sweeps (MgSel::halves half-sweeps, in place in the
//          stage, the first of MgSel::colour), from zero or from the level's values
// A step alone is a launch that waits for its work list, its brick's neighbours and one stage: 4 to
// 9 us however small the level, 24 us a sweep at the finest level of 3.1k bricks, most of it latency.
enum Leg { REST = 0, DOWN = 1, UP = 2, PUP = 3, RB = 4 };
constexpr int rimOf(int leg) { return leg == RB ? 4 : 3; }

// Legs may be launched while the one before still runs (MgSel::overlap, fp_overlap.cuh): a leg lets its
// successor start at once, and waits for its predecessor where it first reads what that wrote. What it
// reads before then (parameters, lists, records) was complete before the kernel ahead of the first of
// the legs started.
// A staged cell's flags: 0 for no unknown (its value becomes zero), else one of
constexpr uint8_t RIM_OPEN = 0x80;   // an unknown, not solid: the sweeps update it (bits 0-5: its open sides)
constexpr uint8_t RIM_SOLID = 0x01;  // an unknown that is solid: zero too

// The shapes: OWN cells a side, pieces of 4 values (16 bytes, or 8 in BF16) a row: one before, one
// after, so that every piece lies in one owner's row.
template <int OWN, int RIM>
struct Rim {
  static constexpr int R = RIM, S = OWN + 2 * R;     // the box of values and flags
  static constexpr int PIECES = OWN / 4 + 2, P = OWN == 8 ? 20 : 12;  // a row's pieces; its pitch (bank spread)
  static constexpr int C = S - 2;                    // the box the first sweep covers, and the right-hand sides'
  static constexpr int H = OWN / 2, G = H + 4;       // the level below: cells a side, and with a rim of two
  static constexpr int THREADS = OWN == 8 ? 256 : 128;
  static constexpr int VALUES = S * S * P, SWEPT = C * C * P;
  static constexpr int OTHER = R == 4 ? 0 : SWEPT, BELOW = R == 4 ? 0 : G * G * G;  // red-black works in place
  static constexpr size_t SMEM = (VALUES + SWEPT + OTHER + BELOW) * sizeof(float) + VALUES;
};
// The shared memory of a box, carved.
template <int OWN, int R>
struct RimStage {
  float *val, *rh, *other, *below;
  uint8_t* fl;
  FP_DEV explicit RimStage(float* smem) {
    using K = Rim<OWN, R>;
    val = smem;
    rh = val + K::VALUES;
    other = rh + K::SWEPT;
    below = other + K::OTHER;
    fl = reinterpret_cast<uint8_t*>(below + K::BELOW);
  }
  // The place of cell (x,y,z), from the owner's first, among the values and flags; among the rest.
  FP_DEV static int at(int x, int y, int z) { return ((z + R) * Rim<OWN, R>::S + y + R) * Rim<OWN, R>::P + x + 4; }
  FP_DEV static int in(int x, int y, int z) { return ((z + R - 1) * Rim<OWN, R>::C + y + R - 1) * Rim<OWN, R>::P + x + 4; }
};

// Four, or two, values of a level from index a.
FP_DEV float4 ld4(const float* p, long a, bool narrow) {
  if (!narrow) return *reinterpret_cast<const float4*>(p + a);
  const __nv_bfloat162* q = reinterpret_cast<const __nv_bfloat162*>(reinterpret_cast<const __nv_bfloat16*>(p) + a);
  const float2 u = __bfloat1622float2(q[0]), v = __bfloat1622float2(q[1]);
  return make_float4(u.x, u.y, v.x, v.y);
}
FP_DEV float2 ld2(const float* p, long a, bool narrow) {
  if (!narrow) return *reinterpret_cast<const float2*>(p + a);
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(reinterpret_cast<const __nv_bfloat16*>(p) + a));
}
FP_DEV uint8_t rimFlag(uint8_t topo, bool unknown) {
  return (uint8_t)(!unknown ? 0u : ((topo & FP_STORED_SOLID) ? RIM_SOLID : (RIM_OPEN | (topo & 63u))));
}

// Fill the stage of the box of an owner of OWN^3 cells whose 27 neighbours' storage is nbr[] (their
// slots, -1 none), RV cells out for values, RR for right-hand sides, RF for flags: from `topo` and
// `open(n, low, cell)`, whether cell `cell` of neighbour n, on its low faces on the axes of bits
// `low`, is an unknown.
template <int RV, int RR, int RF, int OWN, int R, class Open>
FP_DEV void stageRim(const RimStage<OWN, R>& st, const int* nbr, const Args& A, const uint8_t* topo, Open open) {
  using K = Rim<OWN, R>;
  constexpr int M = OWN - 1, CELLS = OWN * OWN * OWN, E = OWN + 2 * RV;
  static_assert(RV >= RR && RV >= RF, "the values' box holds the others");
  for (int i = threadIdx.x; i < E * E * K::PIECES; i += K::THREADS) {
    const int piece = i % K::PIECES, row = i / K::PIECES, y = row % E - RV, z = row / E - RV;
    const int dx = piece == 0 ? -1 : (piece == K::PIECES - 1 ? 1 : 0), dy = y < 0 ? -1 : (y >= OWN ? 1 : 0),
              dz = z < 0 ? -1 : (z >= OWN ? 1 : 0);
    const int n = nbrIndex(dx, dy, dz), s = nbr[n], x = piece * 4 - 4;
    const int cell = ((z & M) * OWN + (y & M)) * OWN + (x & M);
    const long at = (long)s * CELLS + cell;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s >= 0 && (R != 4 || A.pin)) v = ld4(A.pin, at, A.pinN);
    *reinterpret_cast<float4*>(st.val + st.at(x, y, z)) = v;
    auto within = [&](int r) { return y >= -r && y < OWN + r && z >= -r && z < OWN + r; };
    if (within(RR)) {
      float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s >= 0) r = ld4(A.rhs, at, A.rhsN);
      *reinterpret_cast<float4*>(st.rh + st.in(x, y, z)) = r;
    }
    if (within(RF)) {
      uchar4 f = make_uchar4(0, 0, 0, 0);
      if (s >= 0) {
        const uchar4 t = *reinterpret_cast<const uchar4*>(topo + at);
        const unsigned low = ((y & M) == 0 ? 2u : 0u) | ((z & M) == 0 ? 4u : 0u);
        // The piece before the row starts on no low face that flags are asked of (OWN > RF).
        const unsigned edge = ((x & M) == 0 && dx >= 0) ? low | 1u : low;
        f = make_uchar4(rimFlag(t.x, open(n, edge, cell)), rimFlag(t.y, open(n, low, cell + 1)),
                        rimFlag(t.z, open(n, low, cell + 2)), rimFlag(t.w, open(n, low, cell + 3)));
      }
      *reinterpret_cast<uchar4*>(st.fl + st.at(x, y, z)) = f;
    }
  }
}
// The level below around the owner, a rim of two, as prolongation reads it: coarseValue of every
// cell. `below(c, n)` gives a cell's index in the level's storage (-1 none) from its neighbour n and
// its place there; a solid cell's ghost comes through the directory (few cells, near colliders).
template <int OWN, int R, class Below>
FP_DEV void stageBelow(const SimParams& P, const Home& H, const RimStage<OWN, R>& st, const Args& A, int bx, int by, int bz,
                       Below below) {
  using K = Rim<OWN, R>;
  for (int i = threadIdx.x; i < K::G * K::G * K::G; i += K::THREADS) {
    const int x = i % K::G - 2, y = i / K::G % K::G - 2, z = i / (K::G * K::G) - 2;
    const int dx = x < 0 ? -1 : (x >= K::H ? 1 : 0), dy = y < 0 ? -1 : (y >= K::H ? 1 : 0), dz = z < 0 ? -1 : (z >= K::H ? 1 : 0);
    const long a = below(nbrIndex(dx, dy, dz), ((z & (K::H - 1)) * K::H + (y & (K::H - 1))) * K::H + (x & (K::H - 1)));
    float v = 0.f;
    if (a >= 0)
      v = (P.colliderCount > 0 && (P.topo[A.level + 1][a] & FP_STORED_SOLID)) 
              ? coarseValue(P, H, A.coarse, A.level + 1, bx + x, by + y, bz + z)
              : ldBf(A.coarse, a, A.coarseN);
    st.below[i] = v;
  }
}
// prolongCell of the box, in place; `groundRow`: the lowest row of the level below that is not below
// the ground (its ghosts mirror the ground).
template <int OWN, int R>
FP_DEV void prolongRim(const RimStage<OWN, R>& st, int groundRow, bool narrow) {
  using K = Rim<OWN, R>;
  for (int i = threadIdx.x; i < K::S * K::S * K::S; i += K::THREADS) {
    const int x = i % K::S - K::R, y = i / K::S % K::S - K::R, z = i / (K::S * K::S) - K::R, o = st.at(x, y, z);
    float v = 0.f;
    if (st.fl[o] & RIM_OPEN) {
      // Cell p lies a quarter of a coarse cell past centre (p - 1) >> 1 when odd, three when even.
      const int ix = ((x - 1) >> 1) + 2, iz = ((z - 1) >> 1) + 2;
      const int iy[2] = {min(max((y - 1) >> 1, groundRow) + 2, K::G - 1), min(max(((y - 1) >> 1) + 1, groundRow) + 2, K::G - 1)};
      const float fx = (x & 1) ? 0.25f : 0.75f, fy = (y & 1) ? 0.25f : 0.75f, fz = (z & 1) ? 0.25f : 0.75f;
      float c[8];
#pragma unroll
      for (int k = 0; k < 8; k++) c[k] = st.below[((iz + (k >> 2)) * K::G + iy[(k >> 1) & 1]) * K::G + ix + (k & 1)];
      const float corr = mixf(mixf(mixf(c[0], c[1], fx), mixf(c[2], c[3], fx), fy),
                              mixf(mixf(c[4], c[5], fx), mixf(c[6], c[7], fx), fy), fz);
      v = st.val[o] + corr;
      if (narrow) v = __bfloat162float(__float2bfloat16_rn(v));
    }
    st.val[o] = v;
  }
}

// One sweep over the box RIM cells around the owner's cells, from `in` (whose cell (x,y,z) is at
// place(x,y,z), its rows SZ a layer).
template <int RIM, int SZ, int OWN, int R, class Place, class Put>
FP_DEV void sweepBox(const RimStage<OWN, R>& st, const float* in, Place place, bool narrow, Put put) {
  using K = Rim<OWN, R>;
  constexpr int E = OWN + 2 * RIM;
  for (int i = threadIdx.x; i < E * E * E; i += K::THREADS) {
    const int x = i % E - RIM, y = i / E % E - RIM, z = i / (E * E) - RIM;
    const int c = place(x, y, z);
    const uint32_t f = st.fl[st.at(x, y, z)];
    float v = 0.f;
    if (f & RIM_OPEN) {
      constexpr int sy = K::P, sz = SZ * K::P;
      const float v0 = (f & 1u) ? in[c + 1] : 0.f, v1 = (f & 2u) ? in[c - 1] : 0.f;
      const float v2 = (f & 4u) ? in[c + sy] : 0.f, v3 = (f & 8u) ? in[c - sy] : 0.f;
      const float v4 = (f & 16u) ? in[c + sz] : 0.f, v5 = (f & 32u) ? in[c - sz] : 0.f;
      const float sum = (v0 + v1) + (v2 + v3) + (v4 + v5);
      const float cand = (sum - st.rh[st.in(x, y, z)]) / fmaxf(diagOf(f & 63u), 1e-12f);
      v = mixf(in[c], cand, 0.8f);
      if (narrow) v = __bfloat162float(__float2bfloat16_rn(v));
    }
    put(x, y, z, v);
  }
}
// A red-black half-sweep over the box RIM cells around the owner's, in place: relaxCell's red-black branch,
// the colour's other cells not touched. The box's last half-sweep is that of RIM 0, so this is the one
// before it RIM times; nothing where the launch has fewer.
template <int RIM, int OWN, int R>
FP_DEV void halfSweep(const RimStage<OWN, R>& st, const Args& A) {
  using K = Rim<OWN, R>;
  constexpr int E = OWN + 2 * RIM, HALF = E / 2, sy = K::P, sz = K::S * K::P;
  if (A.halves <= RIM) return;  // the same for the whole CTA
  const int colour = (A.colour - 1 + A.halves - 1 - RIM) & 1;
  for (int i = threadIdx.x; i < E * E * HALF; i += K::THREADS) {
    const int row = i / HALF, y = row % E - RIM, z = row / E - RIM;
    // An owner's first cell is even on each axis: the colour's cells of a row from its first or second.
    const int x = i % HALF * 2 - RIM + ((colour + RIM + y + z) & 1);
    const int c = st.at(x, y, z);
    const uint32_t f = st.fl[c];
    float v = 0.f;
    if (f & RIM_OPEN) {
      const float v0 = (f & 1u) ? st.val[c + 1] : 0.f, v1 = (f & 2u) ? st.val[c - 1] : 0.f;
      const float v2 = (f & 4u) ? st.val[c + sy] : 0.f, v3 = (f & 8u) ? st.val[c - sy] : 0.f;
      const float v4 = (f & 16u) ? st.val[c + sz] : 0.f, v5 = (f & 32u) ? st.val[c - sz] : 0.f;
      const float sum = (v0 + v1) + (v2 + v3) + (v4 + v5);
      v = (sum - st.rh[st.in(x, y, z)]) / fmaxf(diagOf(f & 63u), 1e-12f);
      if (A.poutN) v = __bfloat162float(__float2bfloat16_rn(v));
    }
    st.val[c] = v;
  }
  __syncthreads();
}
// The leg on a staged box; `own(cell, value)` takes the owner's results. DOWN leaves them (and a rim of
// one) in st.val at st.in for the restriction.
template <int LEG, int OWN, int R, class Own>
FP_DEV void sweepRim(const RimStage<OWN, R>& st, const Args& A, Own own) {
  using K = Rim<OWN, R>;
  const bool narrow = A.poutN;
  if constexpr (LEG == REST) return;
  if constexpr (LEG == RB) {
    halfSweep<3>(st, A);
    halfSweep<2>(st, A);
    halfSweep<1>(st, A);
    halfSweep<0>(st, A);
    for (int c = threadIdx.x; c < OWN * OWN * OWN; c += K::THREADS)
      own(c, st.val[st.at(c % OWN, c / OWN % OWN, c / (OWN * OWN))]);
    return;
  }
  auto at = [&](int x, int y, int z) { return st.at(x, y, z); };
  auto in = [&](int x, int y, int z) { return st.in(x, y, z); };
  auto cell = [](int x, int y, int z) { return (z * OWN + y) * OWN + x; };
  sweepBox<2, K::S>(st, st.val, at, narrow, [&](int x, int y, int z, float v) { st.other[st.in(x, y, z)] = v; });
  __syncthreads();
  sweepBox<1, K::C>(st, st.other, in, narrow, [&](int x, int y, int z, float v) {
    st.val[st.in(x, y, z)] = v;
    if (LEG == DOWN && x >= 0 && x < OWN && y >= 0 && y < OWN && z >= 0 && z < OWN) own(cell(x, y, z), v);
  });
  __syncthreads();
  if constexpr (LEG == UP || LEG == PUP)
    sweepBox<0, K::C>(st, st.val, in, narrow, [&](int x, int y, int z, float v) { own(cell(x, y, z), v); });
}
// restrictCell of coarse cell q of the owner's (OWN / 2)^3 from the values after DOWN's sweeps, or as
// staged; whether all its cells are unknowns.
template <int LEG, int OWN, int R>
FP_DEV float restrictRim(const RimStage<OWN, R>& st, int q, bool& every) {
  using K = Rim<OWN, R>;
  const int cx = q % K::H, cy = q / K::H % K::H, cz = q / (K::H * K::H);
  constexpr int sy = K::P, sz = (LEG == DOWN ? K::C : K::S) * K::P;
  float residual = 0.f;
  every = true;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int x = cx * 2 + (k & 1), y = cy * 2 + ((k >> 1) & 1), z = cz * 2 + (k >> 2);
    const int o = LEG == DOWN ? st.in(x, y, z) : st.at(x, y, z);
    const uint32_t f = st.fl[st.at(x, y, z)];
    every = every && f != 0u;
    if (f & RIM_OPEN) {
      const float v0 = (f & 1u) ? st.val[o + 1] : 0.f, v1 = (f & 2u) ? st.val[o - 1] : 0.f;
      const float v2 = (f & 4u) ? st.val[o + sy] : 0.f, v3 = (f & 8u) ? st.val[o - sy] : 0.f;
      const float v4 = (f & 16u) ? st.val[o + sz] : 0.f, v5 = (f & 32u) ? st.val[o - sz] : 0.f;
      const float sum = (v0 + v1) + (v2 + v3) + (v4 + v5);
      residual += st.rh[st.in(x, y, z)] - (sum - diagOf(f & 63u) * st.val[o]);
    }
  }
  return residual * 0.5f;
}
// What the restriction writes of coarse cell `out` of the level below.
FP_DEV void storeCoarse(const SimParams& P, const Args& A, long out, float r, bool every) {
  stBf(const_cast<float*>(A.coarse), out, r, A.coarseN);  // the coarse right-hand side
  float first = 0.f;
  if (every) {
    const uint32_t f = expandFlags(P.topo[A.level + 1][out]);
    if (!(f & SOLIDF)) first = mixf(0.f, (0.f - r) / fmaxf(diagOf(f), 1e-12f), 0.8f);
  }
  stBf(A.cfirst, out, first, A.cfirstN);
}
template <int LEG, int OWN, int R, class Open>
FP_DEV void stageLeg(const RimStage<OWN, R>& st, const int* nbr, const Args& A, const uint8_t* topo, Open open) {
  if constexpr (LEG == REST)
    stageRim<1, 0, 0>(st, nbr, A, topo, open);
  else if constexpr (LEG == RB)
    stageRim<4, 3, 3>(st, nbr, A, topo, open);
  else if constexpr (LEG == PUP)
    stageRim<3, 2, 3>(st, nbr, A, topo, open);
  else
    stageRim<3, 2, 2>(st, nbr, A, topo, open);
}
// activeCell on a brick level: a cell is an unknown when its brick and those before it on the axes of
// its low faces compute. Bit n of `ok`: neighbour n does, or lies below the ground (not asked).
FP_DEV bool openIn(uint32_t ok, int n, unsigned low) {
  uint32_t need = 1u << n;
  if (low & 1u) need |= need >> 1;
  if (low & 2u) need |= need >> 3;
  if (low & 4u) need |= need >> 9;
  return (ok & need) == need;
}
FP_DEV int groundRowOf(const SimParams& P, int firstRow) { return P.ground ? -firstRow : -(1 << 20); }

// Brick levels of OWN^3 cells a brick (8 or 4), a CTA a brick. A.pin: the level's values; A.pout: the
// result, the other buffer; REST, DOWN: A.coarse the coarse right-hand side, A.cfirst its first
// iterate; PUP: A.coarse the level below.
template <int OWN, int LEG>
__global__ void __launch_bounds__(Rim<OWN, rimOf(LEG)>::THREADS) k_leg_bricks(FpBatch bt, MgSel Sl) {
  using K = Rim<OWN, rimOf(LEG)>;
  __shared__ int nslot[27];
  __shared__ uint32_t okBits;
  extern __shared__ __align__(16) float rimSmem[];
  const RimStage<OWN, K::R> st(rimSmem);
  const int t = threadIdx.x;
  letNextStart();
  const uint32_t total = workTotal(bt, FP_WORK_ACTIVE);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t i;
    const SimParams& P = *workSim(bt, FP_WORK_ACTIVE, item, i).vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    const uint32_t id = P.active[i];
    if (!homeOk(P, id)) continue;  // the bounds-checked build only
    const Home H = homeOf(P, id, nslot);
    __syncthreads();  // the previous brick's stage has been read
    if (t < 32) {
      bool ok = false;
      if (t < 27) {
        const int s = checkSlot(P, FP_SITE_RECORD, entryPage(P.records[(size_t)id * FP_RECORD_WORDS + t]));
        nslot[t] = s;
        ok = s >= 0 || (P.ground && H.by + (t / 3) % 3 - 1 < 0);
      }
      const uint32_t b = __ballot_sync(0xffffffffu, ok);
      if (t == 0) okBits = b;
    }
    __syncthreads();
    const uint32_t ok = okBits;
    waitForPrevious();
    stageLeg<LEG>(st, nslot, A, P.topo[A.level], [&](int n, unsigned low, int) { return openIn(ok, n, low); });
    if constexpr (LEG == PUP) {
      stageBelow(P, H, st, A, H.bx * K::H, H.by * K::H, H.bz * K::H,
                      [&](int n, int c) { return nslot[n] < 0 ? -1l : (long)nslot[n] * (K::H * K::H * K::H) + c; });
      __syncthreads();
      prolongRim(st, groundRowOf(P, H.by * K::H), A.poutN);
    }
    __syncthreads();
    const long slot = nslot[13];
    constexpr int CELLS = OWN * OWN * OWN;
    sweepRim<LEG>(st, A, [&](int c, float v) { stBf(A.pout, slot * CELLS + c, v, A.poutN); });
    if constexpr (LEG == DOWN || LEG == REST)
      for (int q = t; q < CELLS / 8; q += K::THREADS) {
        bool every;
        const float r = restrictRim<LEG>(st, q, every);
        storeCoarse(P, A, slot * (CELLS / 8) + q, r, every);
      }
  }
  waitForPrevious();
}

// The first tile level (4^3 cells a tile, a cell a brick), a CTA a live tile (a neighbour tile that
// exists is live).
template <int LEG>
__global__ void __launch_bounds__(Rim<4, rimOf(LEG)>::THREADS) k_leg_tiles(FpBatch bt, MgSel Sl) {
  using K = Rim<4, rimOf(LEG)>;
  __shared__ int nbr[27];
  __shared__ uint64_t masks[27];
  extern __shared__ __align__(16) float rimSmem[];
  const RimStage<4, K::R> st(rimSmem);
  const int t = threadIdx.x;
  letNextStart();
  const uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item, local).vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    const int tile = P.liveTiles[local];
    const int4 rec = __ldg(&P.tileRec[tile]);
    if (rec.w == 0) continue;
    __syncthreads();  // the previous tile's stage has been read
    if (t < 27) {
      const int n = checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[(size_t)tile * 27 + t]));
      nbr[t] = n;
      masks[t] = n >= 0 ? P.tileMask[n] : 0ull;
    }
    __syncthreads();
    waitForPrevious();
    stageLeg<LEG>(st, nbr, A, P.topo[A.level], [&](int n, unsigned, int cell) { return ((masks[n] >> cell) & 1ull) != 0ull; });
    if constexpr (LEG == PUP) {
      const Home H = enterTile(P, tile, rec);
      stageBelow(P, H, st, A, rec.x * K::H, rec.y * K::H, rec.z * K::H,
                    [&](int n, int c) { return nbr[n] < 0 ? -1l : (long)nbr[n] * 8 + c; });
      __syncthreads();
      prolongRim(st, groundRowOf(P, rec.y * K::H), A.poutN);
    }
    __syncthreads();
    sweepRim<LEG>(st, A, [&](int c, float v) { stBf(A.pout, (long)tile * 64 + c, v, A.poutN); });
    if (LEG == DOWN && t < 8) {
      bool every;
      const float r = restrictRim<LEG>(st, t, every);
      storeCoarse(P, A, (long)tile * 8 + t, r, every);
    }
  }
  waitForPrevious();
}

// The last brick level (2^3 cells a brick), whose three-cell rim reaches past a brick's neighbours: a
// CTA a live tile, the tile's 8^3 cells read and written through its bricks' slots, and those of the
// two bricks around it.
template <int LEG>
__global__ void __launch_bounds__(Rim<8, rimOf(LEG)>::THREADS) k_leg_pairs(FpBatch bt, MgSel Sl) {
  using K = Rim<8, rimOf(LEG)>;
  constexpr int N = 8;  // bricks a side: the tile's four and two on either side
  __shared__ int nbr[27];
  __shared__ int slots[N * N * N];
  __shared__ uint32_t ok[N * N * N / 32];
  extern __shared__ __align__(16) float rimSmem[];
  const RimStage<8, K::R> st(rimSmem);
  const int t = threadIdx.x;
  letNextStart();
  const uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item, local).vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    const int tile = P.liveTiles[local];
    const int4 rec = __ldg(&P.tileRec[tile]);
    if (rec.w == 0) continue;
    __syncthreads();  // the previous tile's stage has been read
    if (t < 27) nbr[t] = checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[(size_t)tile * 27 + t]));
    __syncthreads();
    for (int i = t; i < N * N * N; i += K::THREADS) {
      const int bx = i % N - 2, by = i / N % N - 2, bz = i / (N * N) - 2;
      const int n = nbr[nbrIndex(bx >> 2, by >> 2, bz >> 2)];
      int s = -1;
      if (n >= 0) s = checkSlot(P, FP_SITE_ENTRY, entryPage(P.entries[(size_t)n * 64 + ((bz & 3) * 4 + (by & 3)) * 4 + (bx & 3)]));
      slots[i] = s;
      const uint32_t b = __ballot_sync(0xffffffffu, s >= 0 || (P.ground && rec.y * 4 + by < 0));
      if ((t & 31) == 0) ok[i >> 5] = b;
    }
    __syncthreads();
    auto okAt = [&](int i) { return ((ok[i >> 5] >> (i & 31)) & 1u) != 0u; };
    waitForPrevious();
    // Pairs of cells along x: a row of the box lies in eight bricks.
    const uint8_t* topo = P.topo[A.level];
    for (int i = t; i < K::S * K::S * N; i += K::THREADS) {
      const int px = i % N, row = i / N, x = px * 2 - 4, y = row % K::S - K::R, z = row / K::S - K::R;
      const int b = (((z >> 1) + 2) * N + (y >> 1) + 2) * N + px, s = slots[b];
      const long at = (long)s * 8 + ((z & 1) * 2 + (y & 1)) * 2;
      float2 v = make_float2(0.f, 0.f), r = v;
      uchar2 f = make_uchar2(0, 0);
      if (s >= 0) {
        if (LEG != RB || A.pin) v = ld2(A.pin, at, A.pinN);
        const uchar2 q = *reinterpret_cast<const uchar2*>(topo + at);
        // The cells of the outermost bricks that a box reaches are on no low face.
        bool in = okAt(b);
        if (!(y & 1) && b >= N) in = in && okAt(b - N);
        if (!(z & 1) && b >= N * N) in = in && okAt(b - N * N);
        if (!(y & 1) && !(z & 1) && b >= N * N + N) in = in && okAt(b - N * N - N);
        bool edge = in;
        if (px > 0) {
          edge = edge && okAt(b - 1);
          if (!(y & 1) && b >= N + 1) edge = edge && okAt(b - N - 1);
          if (!(z & 1) && b >= N * N + 1) edge = edge && okAt(b - N * N - 1);
          if (!(y & 1) && !(z & 1) && b >= N * N + N + 1) edge = edge && okAt(b - N * N - N - 1);
        }
        f = make_uchar2(rimFlag(q.x, edge), rimFlag(q.y, in));
      }
      const int o = st.at(x, y, z);
      *reinterpret_cast<float2*>(st.val + o) = v;
      *reinterpret_cast<uchar2*>(st.fl + o) = f;
      if (y > -K::R && y < 7 + K::R && z > -K::R && z < 7 + K::R) {
        if (s >= 0) r = ld2(A.rhs, at, A.rhsN);
        *reinterpret_cast<float2*>(st.rh + st.in(x, y, z)) = r;
      }
    }
    if constexpr (LEG == PUP) {
      const Home H = enterTile(P, tile, rec);
      stageBelow(P, H, st, A, rec.x * K::H, rec.y * K::H, rec.z * K::H,
                    [&](int n, int c) { return nbr[n] < 0 ? -1l : (long)nbr[n] * 64 + c; });
      __syncthreads();
      prolongRim(st, groundRowOf(P, rec.y * K::H), A.poutN);
    }
    __syncthreads();
    auto slotOf = [&](int bx, int by, int bz) { return slots[((bz + 2) * N + by + 2) * N + bx + 2]; };
    sweepRim<LEG>(st, A, [&](int c, float v) {
      const int x = c & 7, y = (c >> 3) & 7, z = c >> 6, s = slotOf(x >> 1, y >> 1, z >> 1);
      if (s >= 0) stBf(A.pout, (long)s * 8 + ((z & 1) * 2 + (y & 1)) * 2 + (x & 1), v, A.poutN);
    });
    // A coarse cell is a brick's, at the brick's own id; those of bricks without a slot are cleared
    // with the tile masks.
    if (LEG == DOWN && t < 64 && slotOf(t & 3, (t >> 2) & 3, t >> 4) >= 0) {
      bool every;
      const float r = restrictRim<LEG>(st, t, every);
      storeCoarse(P, A, (long)tile * 64 + t, r, every);
    }
  }
  waitForPrevious();
}

// Every cell of `A.level` (a tile level of CELLS cells a tile, 8 or 1) in every tile: a thread per
// cell, 64 / CELLS tiles per CTA; no barriers, so threads of dead tiles just move on.
template <int OP, int CELLS>
__global__ void __launch_bounds__(64) k_level_tiles(FpBatch bt, MgSel Sl) {
  constexpr int NT = 64 / CELLS, s = CELLS == 8 ? 1 : 0, side = 1 << s;
  const int g = threadIdx.x / CELLS, o = threadIdx.x % CELLS;
  uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t item = blockIdx.x * NT + g; item < total; item += gridDim.x * NT) {
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item, local).vview;
    const int t = P.liveTiles[local];
    const Args A = resolve(P, Sl);
    if (A.skip) continue;
    int4 rec = __ldg(&P.tileRec[t]);
    if (rec.w == 0) continue;
    Home H = enterTile(P, t, rec);
    int lx = o & (side - 1), ly = (o >> s) & (side - 1), lz = o >> (2 * s);
    levelCell<OP>(P, H, A, (long)t * CELLS + o, rec.x * side + lx, rec.y * side + ly, rec.z * side + lz);
  }
}

// Staged tile levels: k_level_bricks_staged with a live tile in place of a brick. A group of 64
// threads copies, for its tile, the values of the level it reads over the tile and a rim from
// the tile's 27 neighbour tiles (tileNbr) into shared memory; a cell is an unknown when its
// brick computes (the tile's mask, tileCellActive). Same arithmetic, same order as restrictCell and
// prolongCell. (The first tile level's sweeps are legs.)
//   RESTRICT  stage A.pin at A.level - 1 (TS = 4: the first tile level, a cell a brick); write A.pout, A.cfirst at A.level (2^3 a tile)
//   PROLONG   stage A.coarse at A.level + 1 (TS = 2); write A.pout at A.level (4^3 a tile)
template <int OP, int TS>
struct TileStaged {
  static constexpr int R = OP == PROLONG ? 2 : 1;  // prolongation's Neumann ghosts reach two
  static constexpr int S = TS + 2 * R, S2 = S * S, S3 = S2 * S;
  static constexpr int FS = OP == PROLONG ? 2 * TS : TS;  // the fine level's side (4: a cell a brick)
  static constexpr int FCELLS = FS * FS * FS;
  static constexpr int GROUP = 64, NG = 4;  // threads per tile, tiles per CTA
  static constexpr int WORDS = S3 + (OP == PROLONG ? (S3 + 3) / 4 : 0);  // values + solid bytes
  static constexpr size_t SMEM = (size_t)NG * WORDS * sizeof(float);
  static_assert(FS == 4 && FCELLS == GROUP, "the fine level is the first tile level, a thread a cell");
};

template <int OP, int TS>
__global__ void __launch_bounds__(256) k_level_tiles_staged(FpBatch bt, MgSel Sl) {
  using K = TileStaged<OP, TS>;
  constexpr int S = K::S, S2 = K::S2, S3 = K::S3, R = K::R, GROUP = K::GROUP, NG = K::NG, FCELLS = K::FCELLS;
  constexpr int TS3 = TS * TS * TS;
  __shared__ int nbrAll[NG][27];
  extern __shared__ float stAll[];
  const int g = threadIdx.x / GROUP, t = threadIdx.x % GROUP;
  int* nbr = nbrAll[g];
  float* st = stAll + g * K::WORDS;
  uint8_t* solidSt = reinterpret_cast<uint8_t*>(st + S3);
  const uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t base = blockIdx.x * NG; base < total; base += gridDim.x * NG) {
    const uint32_t item = base + g;
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item < total ? item : base, local).vview;
    const Args A = resolve(P, Sl);
    const int tile = item < total ? P.liveTiles[local] : 0;
    const int4 rec = item < total ? __ldg(&P.tileRec[tile]) : make_int4(0, 0, 0, 0);
    const bool has = item < total && !A.skip && rec.w != 0;
    const int fineLevel = OP == RESTRICT ? A.level - 1 : A.level;
    const int stageLevel = OP == PROLONG ? A.level + 1 : fineLevel;
    const float* src = OP == PROLONG ? A.coarse : A.pin;
    const bool srcN = OP == PROLONG ? A.coarseN : A.pinN;
    if (has && t < 27) nbr[t] = checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[(size_t)tile * 27 + t]));
    __syncthreads();
    // The stage's first cell, in cells of the staged level.
    const int ox = rec.x * TS - R, oy = rec.y * TS - R, oz = rec.z * TS - R;
    // This thread's fine cell (PROLONG): its flags and value, loaded before the stage so that both
    // sets of loads are in flight together.
    const long own = (long)tile * FCELLS + t;
    uint8_t ownTopo = 0;
    float ownValue = 0.f;
    if (OP == PROLONG && has) {
      ownTopo = P.topo[fineLevel][own];
      ownValue = ldBf(A.pin, own, A.pinN);
    }
    bool solidStaged = false;
    if (has) {
      for (int q = t; q < S3; q += GROUP) {
        const int lx = q % S, ly = (q / S) % S, lz = q / S2;
        const int dx = lx < R ? -1 : (lx >= R + TS ? 1 : 0), dy = ly < R ? -1 : (ly >= R + TS ? 1 : 0),
                  dz = lz < R ? -1 : (lz >= R + TS ? 1 : 0);
        const int n = nbr[nbrIndex(dx, dy, dz)];
        const int cx = (lx - R) & (TS - 1), cy = (ly - R) & (TS - 1), cz = (lz - R) & (TS - 1);
        const long a = n < 0 ? -1 : (long)n * TS3 + (cz * TS + cy) * TS + cx;
        st[q] = a < 0 ? 0.f : ldBf(src, a, srcN);
        if (OP == PROLONG) {
          const bool solid = a >= 0 && (P.topo[stageLevel][a] & FP_STORED_SOLID);
          solidSt[q] = solid ? 1 : 0;
          solidStaged = solidStaged || solid;
        }
      }
    }
    bool anySolid = false;
    if (OP == PROLONG)
      anySolid = __syncthreads_or(solidStaged) != 0;
    else
      __syncthreads();
    if (has) {
      const uint64_t mask = P.tileMask[tile];
      auto unknown = [&](int lx, int ly, int lz) { return ((mask >> ((lz * 4 + ly) * 4 + lx)) & 1ull) != 0ull; };
      auto sumAt = [&](int lx, int ly, int lz, uint32_t f) {
        int c = ((lz + 1) * S + (ly + 1)) * S + (lx + 1);
        float v0 = (f & 1u) ? st[c + 1] : 0.f, v1 = (f & 2u) ? st[c - 1] : 0.f;
        float v2 = (f & 4u) ? st[c + S] : 0.f, v3 = (f & 8u) ? st[c - S] : 0.f;
        float v4 = (f & 16u) ? st[c + S2] : 0.f, v5 = (f & 32u) ? st[c - S2] : 0.f;
        return (v0 + v1) + (v2 + v3) + (v4 + v5);
      };
      const int lx = t & 3, ly = (t >> 2) & 3, lz = t >> 4;
      const int px = rec.x * 4 + lx, py = rec.y * 4 + ly, pz = rec.z * 4 + lz;
      if (OP == PROLONG) {
        const uint32_t f = expandFlags(ownTopo);
        if ((f & SOLIDF) || !unknown(lx, ly, lz)) {
          stBf(A.pout, own, 0.f, A.poutN);
        } else {
          float qx = ((float)px + 0.5f) * 0.5f - 0.5f, qy = ((float)py + 0.5f) * 0.5f - 0.5f,
                qz = ((float)pz + 0.5f) * 0.5f - 0.5f;
          int ix = (int)floorf(qx), iy = (int)floorf(qy), iz = (int)floorf(qz);
          float fx = qx - floorf(qx), fy = qy - floorf(qy), fz = qz - floorf(qz);
          bool fast = (P.colliderCount == 0 || !anySolid) && (!P.ground || iy >= 0);
          // Below the ground the mirrored ghosts read the row above it, which a tile under y = 0
          // does not stage: those read through the directory.
          const bool staged = !(P.ground && rec.y < 0);
          auto at = [&](int x, int y, int z) { return ((z - oz) * S + (y - oy)) * S + (x - ox); };
          auto ghost = [&](int cx, int cy, int cz) {
            int groundY = P.ground ? 0 : -0x7fffffff;
            int c[3] = {cx, max(cy, groundY), cz};
            int ci = at(c[0], c[1], c[2]);
            if (!solidSt[ci]) return st[ci];
            float sum = 0.f, count = 0.f;
            for (int axis = 0; axis < 3; axis++)
              for (int side = -1; side <= 1; side += 2) {
                int q[3] = {c[0], c[1], c[2]};
                q[axis] += side;
                q[1] = max(q[1], groundY);
                int qi = at(q[0], q[1], q[2]);
                if (!solidSt[qi]) {
                  sum += st[qi];
                  count += 1.f;
                }
              }
            return sum / fmaxf(count, 1.f);
          };
          float v[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
            if (fast) {
              v[q] = st[at(ix + dx, iy + dy, iz + dz)];
            } else if (staged) {
              v[q] = ghost(ix + dx, iy + dy, iz + dz);
            } else {
              Home H = enterTile(P, tile, rec);
              v[q] = coarseValue(P, H, A.coarse, A.level + 1, ix + dx, iy + dy, iz + dz);
            }
          }
          float corr = mixf(mixf(mixf(v[0], v[1], fx), mixf(v[2], v[3], fx), fy),
                            mixf(mixf(v[4], v[5], fx), mixf(v[6], v[7], fx), fy), fz);
          stBf(A.pout, own, ownValue + corr, A.poutN);
        }
      } else if (t < 8) {  // RESTRICT: the tile's 2^3 coarse cells at A.level
        const int cx = t & 1, cy = (t >> 1) & 1, cz = t >> 2;
        float residual = 0.f;
        bool every = true;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          int fx = cx * 2 + (k & 1), fy = cy * 2 + ((k >> 1) & 1), fz = cz * 2 + (k >> 2);
          bool u = unknown(fx, fy, fz);
          every = every && u;
          if (u) {
            long a = (long)tile * FCELLS + ((fz * 4 + fy) * 4 + fx);
            uint32_t f = expandFlags(P.topo[fineLevel][a]);
            if (!(f & SOLIDF)) {
              float center = st[((fz + 1) * S + (fy + 1)) * S + (fx + 1)];
              residual += ldBf(A.rhs, a, A.rhsN) - (sumAt(fx, fy, fz, f) - diagOf(f) * center);
            }
          }
        }
        float r = residual * 0.5f;
        const long out = (long)tile * 8 + t;
        stBf(A.pout, out, r, A.poutN);
        float first = 0.f;
        if (every) {
          uint32_t f = expandFlags(P.topo[A.level][out]);
          if (!(f & SOLIDF)) first = mixf(0.f, (0.f - r) / fmaxf(diagOf(f), 1e-12f), 0.8f);
        }
        stBf(A.cfirst, out, first, A.cfirstN);
      }
    }
    __syncthreads();
  }
}

// relaxCoarse (pressure.wgsl:549-599): the bottom level, one cell per tile slot, every
// iteration in one CTA; a CTA per simulation. The live tiles stride over the threads. When 28
// bytes a live tile fit `smemBytes`, each one's flags (SOLIDF where it is no unknown),
// right-hand side, face neighbours (as live positions) and a ping-pong pair of values live in
// shared memory; else the values ping-pong between the level's two pressure buffers in global
// memory by slot (same arithmetic, same order).
__global__ void __launch_bounds__(1024) k_bottom(FpBatch bt, MgSel Sl, int iterations, int smemBytes) {
  extern __shared__ float bottomSmem[];
  const int nbIndex[6] = {nbrIndex(1, 0, 0), nbrIndex(-1, 0, 0), nbrIndex(0, 1, 0),
                          nbrIndex(0, -1, 0), nbrIndex(0, 0, 1), nbrIndex(0, 0, -1)};
  int sims = batchCount(bt);
  for (int sim = blockIdx.x; sim < sims; sim += gridDim.x) {
    const SimParams& P = *bt.sims[sim].vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    const int level = A.level, L = P.liveCount;
    auto flagOf = [&](int t) -> uint32_t {  // t is live
      int4 rec = __ldg(&P.tileRec[t]);
      Home H = enterTile(P, t, rec);
      return (activeCell(P, H, rec.x, rec.y, rec.z, level) ? expandFlags(P.topo[level][t]) : SOLIDF) | 0x80000000u;
    };
    if ((long)L * 28 <= (long)smemBytes) {
      float* cur = bottomSmem;
      float* nxt = cur + L;
      float* rhs = nxt + L;
      uint32_t* flags = reinterpret_cast<uint32_t*>(rhs + L);
      int16_t* nb = reinterpret_cast<int16_t*>(flags + L);  // 6 a tile
      for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const int t = P.liveTiles[j];
        const uint32_t f = flagOf(t);
        flags[j] = f;
        rhs[j] = ldBf(A.rhs, t, A.rhsN);
        for (int k = 0; k < 6; k++) {
          int n = ((f >> k) & 1u) ? checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[t * 27 + nbIndex[k]])) : -1;
          nb[j * 6 + k] = (int16_t)(n >= 0 ? P.tileIndex[n] : -1);
        }
        // Cells that are no unknown are never read and become zero in the first iteration.
        cur[j] = !(f & SOLIDF) ? ldBf(A.pin, t, A.pinN) : 0.f;
      }
      __syncthreads();
      for (int it = 0; it < iterations; it++) {
        for (int j = threadIdx.x; j < L; j += blockDim.x) {
          const uint32_t f = flags[j];
          float next = 0.f;
          if (!(f & SOLIDF)) {
            float w[6];
#pragma unroll
            for (int k = 0; k < 6; k++) {
              const int n = nb[j * 6 + k];
              w[k] = n >= 0 ? cur[n] : 0.f;
            }
            float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
            float cand = (sum - rhs[j]) / fmaxf(diagOf(f & 63u), 1e-12f);
            next = mixf(cur[j], cand, 0.8f);
          }
          nxt[j] = next;
        }
        __syncthreads();
        float* tmp = cur;
        cur = nxt;
        nxt = tmp;
      }
      for (int j = threadIdx.x; j < L; j += blockDim.x) stBf(A.pout, P.liveTiles[j], cur[j], A.poutN);
      __syncthreads();
      continue;
    }
    // In global memory: cur starts in pout (a copy of pin), nxt is pin's buffer; both hold the
    // level's storage type.
    float* cur = A.pout;
    float* nxt = const_cast<float*>(A.pin);
    const bool gN = A.poutN;
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
      const int t = P.liveTiles[j];
      const uint32_t f = flagOf(t);
      // pin and pout are the level's two buffers: the copy into pout reads no value it wrote.
      stBf(cur, t, !(f & SOLIDF) ? ldBf(A.pin, t, A.pinN) : 0.f, gN);
    }
    __syncthreads();
    for (int it = 0; it < iterations; it++) {
      for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const int t = P.liveTiles[j];
        const uint32_t f = flagOf(t);
        float next = 0.f;
        if (!(f & SOLIDF)) {
          float w[6];
#pragma unroll
          for (int k = 0; k < 6; k++) {
            int n = ((f >> k) & 1u) ? checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[t * 27 + nbIndex[k]])) : -1;
            w[k] = n >= 0 ? ldBf(cur, n, gN) : 0.f;
          }
          float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
          float cand = (sum - ldBf(A.rhs, t, A.rhsN)) / fmaxf(diagOf(f & 63u), 1e-12f);
          next = mixf(ldBf(cur, t, gN), cand, 0.8f);
        }
        stBf(nxt, t, next, gN);
      }
      __syncthreads();
      float* tmp = cur;
      cur = nxt;
      nxt = tmp;
    }
    if (cur != A.pout)
      for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const int t = P.liveTiles[j];
        stBf(A.pout, t, ldBf(cur, t, gN), A.poutN);
      }
    __syncthreads();
  }
}

// A value as the storage of a level rounds it.
FP_DEV float bfRound(float v, bool narrow) { return narrow ? __bfloat162float(__float2bfloat16_rn(v)) : v; }

// The second tile level (2^3 cells a tile) and the bottom (one cell a tile) in one CTA per
// simulation: the V-cycle from level bl + 1 down (two relaxations, restriction to the bottom,
// the bottom's iterations, prolongation, three relaxations), with both levels' iterates,
// right-hand sides and flags in shared memory by live tile, __syncthreads between sweeps.
// The arithmetic and its order are those of k_level_tiles (relaxCell, restrictCell,
// prolongCell) and k_bottom; every value a level stores is rounded as its storage rounds it.
//   A.level: level bl + 1; A.rhs its right-hand side; A.pin its first iterate; A.pout where
//   its result goes; A.cfirst: the bottom's result (read back by the prolongation).
constexpr int COARSE_SLOT_BYTES = 8 * 3 * 4 + 8 + 3 * 4 + 4 + 6 * 2 + 27 * 2;  // per live tile
constexpr int COARSE_SMEM = 224 * 1024;
constexpr uint32_t LIVE = 0x80000000u, ODD = 0x40000000u;  // a bottom cell's flags: a live tile's; of odd colour
constexpr uint8_t UNKNOWN = 0x80;  // level bl + 1 flag byte: activeCell; bit 6 solid; 0-5 open

// The level bl + 1 cell next to cell o of tile t on side k (+x, -x, +y, -y, +z, -z), as an
// index of the level's tile-slot arrays; -1 without a tile there.
// `faces` holds each live tile's six face neighbours as live positions (-1 without one). Either way
// the cell's place in its tile is o with the axis' bit turned.
FP_DEV int coarseNbr(const int16_t* faces, int j, int o, int k) {
  const int ax = k >> 1, nj = ((o >> ax) & 1) == (k & 1) ? j : faces[j * 6 + k];
  return nj < 0 ? -1 : nj * 8 + (o ^ (1 << ax));
}

// RB: the red-black V-cycle from there down, `pre` sweeps from zero, restriction, `iterations` sweeps of the
// bottom from zero, prolongation, `post` sweeps (odd cells first), in place; the arithmetic of
// k_level_tiles and k_bottom_rb. As a launch a half-sweep it was 107 us of each V-cycle of 2.3k bricks, now 33.
template <bool RB>
__global__ void __launch_bounds__(1024) k_coarse(FpBatch bt, MgSel Sl, int iterations, int smemBytes, int pre, int post) {
  extern __shared__ float coarseSmem[];
  letNextStart();
  const int nbIndex[6] = {nbrIndex(1, 0, 0), nbrIndex(-1, 0, 0), nbrIndex(0, 1, 0),
                          nbrIndex(0, -1, 0), nbrIndex(0, 0, 1), nbrIndex(0, 0, -1)};
  const int sims = batchCount(bt);
  for (int sim = blockIdx.x; sim < sims; sim += gridDim.x) {
    const SimParams& P = *bt.sims[sim].vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    // Shared arrays by live position j (tile slot P.liveTiles[j]); level L cells at j * 8 + o.
    const int L = A.level, BL = L + 1, nt = P.liveCount, n4 = nt * 8;
    if ((long)nt * COARSE_SLOT_BYTES > smemBytes) continue;  // the host sizes launches to fit
    const bool nL = narrowLevel(P, L), nB = narrowLevel(P, BL);
    float* pa = coarseSmem;  // level L: iterates, right-hand side
    float* pb = pa + n4;
    float* rh = pb + n4;
    float* ca = rh + n4;  // bottom: iterates, right-hand side
    float* cb = ca + nt;
    float* cr = cb + nt;
    uint32_t* fb = reinterpret_cast<uint32_t*>(cr + nt);
    uint8_t* fl = reinterpret_cast<uint8_t*>(fb + nt);
    int16_t* faces = reinterpret_cast<int16_t*>(fl + n4);  // six a live tile
    // All 27 neighbour tiles of each live tile: the live position, -2 for a tile that is not
    // live (its stored values are read from global memory), -1 for none.
    int16_t* nb27 = faces + nt * 6;
    bool solidNear = false;  // a bottom cell of a neighbour tile is solid
    // Setting up is chains of dependent loads (a tile, its neighbour, what that holds): several at a
    // time, so that their latencies overlap.
    int* live = reinterpret_cast<int*>(cb);  // until the bottom's iterations
    for (int j = threadIdx.x; j < nt; j += blockDim.x) live[j] = P.liveTiles[j];
    __syncthreads();
    constexpr int AHEAD = 8;
    for (int base = threadIdx.x; base < nt * 27; base += AHEAD * blockDim.x) {
      int n[AHEAD], pos[AHEAD];
      uint8_t tb[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; u++) {
        const int q = base + u * blockDim.x;
        n[u] = q < nt * 27 ? checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[live[q / 27] * 27 + q % 27])) : -1;
      }
#pragma unroll
      for (int u = 0; u < AHEAD; u++) {
        pos[u] = n[u] >= 0 ? P.tileIndex[n[u]] : -1;
        tb[u] = n[u] >= 0 ? P.topo[BL][n[u]] : 0;
      }
#pragma unroll
      for (int u = 0; u < AHEAD; u++) {
        const int q = base + u * blockDim.x;
        if (q >= nt * 27) break;
        const int j = q / 27, k = q % 27;
        nb27[q] = (int16_t)(n[u] < 0 ? -1 : (pos[u] >= 0 ? pos[u] : -2));
        solidNear = solidNear || (tb[u] & FP_STORED_SOLID);
        const int dx = k % 3 - 1, dy = (k / 3) % 3 - 1, dz = k / 9 - 1;
        if ((dx != 0) + (dy != 0) + (dz != 0) == 1) {  // a face: +x, -x, +y, -y, +z, -z
          const int f = dx != 0 ? (dx > 0 ? 0 : 1) : (dy != 0 ? (dy > 0 ? 2 : 3) : (dz > 0 ? 4 : 5));
          faces[j * 6 + f] = (int16_t)pos[u];
        }
      }
    }
    waitForPrevious();
#pragma unroll 4
    for (int c = threadIdx.x; c < n4; c += blockDim.x) {
      const int t = live[c >> 3], o = c & 7;
      const long a = (long)t * 8 + o;  // the cell's storage
      // activeCell of a live tile's own cell: its eight bricks compute (tileCellActive).
      const uint64_t bricks = 0x0000000000330033ull << (2 * (o & 1) + 8 * ((o >> 1) & 1) + 32 * (o >> 2));
      fl[c] = (uint8_t)(P.topo[L][a] | ((P.tileMask[t] & bricks) == bricks ? UNKNOWN : 0));
      pa[c] = RB ? 0.f : ldBf(A.pin, a, nL);
      rh[c] = ldBf(A.rhs, a, nL);
    }
    // Without a solid bottom cell next to any live tile every Neumann ghost of the prolongation
    // is the bottom value itself (coarseValue's first test), read from shared memory.
    const bool anySolid = __syncthreads_or(solidNear) != 0;
    // stencil (pressure.wgsl:360-402) of level L from `src`, cell o of live position j.
    auto sumL = [&](const float* src, int j, int o, uint32_t f) {
      float w[6];
#pragma unroll
      for (int k = 0; k < 6; k++) {
        int n = ((f >> k) & 1u) ? coarseNbr(faces, j, o, k) : -1;
        w[k] = n >= 0 ? src[n] : 0.f;
      }
      return (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
    };
    // relaxCell at level L, src -> dst.
    auto relax = [&](const float* src, float* dst) {
      for (int c = threadIdx.x; c < n4; c += blockDim.x) {
        const uint8_t f = fl[c];
        float v = 0.f;
        if ((f & UNKNOWN) && !(f & FP_STORED_SOLID)) {
          float cand = (sumL(src, c >> 3, c & 7, f & 63u) - rh[c]) / fmaxf(diagOf(f & 63u), 1e-12f);
          v = bfRound(mixf(src[c], cand, 0.8f), nL);
        }
        dst[c] = v;
      }
      __syncthreads();
    };
    // relaxCell's red-black branch at level L, in place: a tile's first cell is even on each axis, so a
    // cell's colour is that of its place in the tile.
    auto half = [&](int colour) {
      for (int i = threadIdx.x; i < nt * 4; i += blockDim.x) {
        const int j = i >> 2, o = (i & 3) * 2 + ((__popc(i & 3) + colour) & 1), c = j * 8 + o;
        const uint8_t f = fl[c];
        float v = 0.f;
        if ((f & UNKNOWN) && !(f & FP_STORED_SOLID))
          v = bfRound((sumL(pa, j, o, f & 63u) - rh[c]) / fmaxf(diagOf(f & 63u), 1e-12f), nL);
        pa[c] = v;
      }
      __syncthreads();
    };
    if constexpr (RB) {
      for (int k = 0; k < pre * 2; k++) half(k & 1);
    } else {
      relax(pa, pb);
      relax(pb, pa);
    }
    // restrictCell into the bottom (one cell a tile), its first iterate and k_bottom's flags.
    for (int j = threadIdx.x; j < nt; j += blockDim.x) {
      const int t = P.liveTiles[j];
      float r = 0.f, first = 0.f;
      uint32_t f = SOLIDF;
      {
        float residual = 0.f;
        bool every = true;
        for (int k = 0; k < 8; k++) {
          const int c = j * 8 + k;
          const uint8_t fk = fl[c];
          every = every && (fk & UNKNOWN);
          if ((fk & UNKNOWN) && !(fk & FP_STORED_SOLID))
            residual += rh[c] - (sumL(pa, j, k, fk & 63u) - diagOf(fk & 63u) * pa[c]);
        }
        r = residual * 0.5f;
        const uint8_t tb = P.topo[BL][t];
        if (every && !(tb & FP_STORED_SOLID)) first = mixf(0.f, (0.f - r) / fmaxf(diagOf(tb & 63u), 1e-12f), 0.8f);
        // activeCell at the bottom covers the tile's 64 bricks: every cell above is an unknown.
        f = (every ? expandFlags(tb) : SOLIDF) | LIVE;
      }
      cr[j] = bfRound(r, nB);
      ca[j] = !RB && !(f & SOLIDF) ? bfRound(first, nB) : 0.f;
      if (RB) {
        const int4 rec = __ldg(&P.tileRec[t]);
        f |= ((rec.x + rec.y + rec.z) & 1) ? ODD : 0u;
      }
      fb[j] = f;
    }
    __syncthreads();
    // relaxCoarse (pressure.wgsl:549-599): FP32 iterates in shared memory.
    float* cur = ca;
    float* nxt = cb;
    // A thread keeps its first tile's flags, neighbours and right-hand side over the iterations (most
    // simulations have a tile a thread at most).
    const int own = threadIdx.x;
    uint32_t ownFlags = SOLIDF;
    float ownRhs = 0.f, ownDiag = 1.f;
    int ownNbr[6] = {-1, -1, -1, -1, -1, -1};
    if (own < nt) {
      ownFlags = fb[own];
      ownRhs = cr[own];
      ownDiag = fmaxf(diagOf(ownFlags & 63u), 1e-12f);
#pragma unroll
      for (int k = 0; k < 6; k++) ownNbr[k] = ((ownFlags >> k) & 1u) ? faces[own * 6 + k] : -1;
    }
    if constexpr (RB) {
      for (int k = 0; k < iterations * 2; k++) {
        if (own < nt && ((ownFlags & ODD) != 0) == ((k & 1) != 0)) {
          float next = 0.f;
          if (!(ownFlags & SOLIDF)) {
            float w[6];
#pragma unroll
            for (int q = 0; q < 6; q++) w[q] = ownNbr[q] >= 0 ? cur[ownNbr[q]] : 0.f;
            const float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
            next = bfRound((sum - ownRhs) / ownDiag, nB);
          }
          cur[own] = next;
        }
        for (int j = own + blockDim.x; j < nt; j += blockDim.x) {
          const uint32_t f = fb[j];
          if (((f & ODD) != 0) != ((k & 1) != 0)) continue;
          float next = 0.f;
          if (!(f & SOLIDF)) {
            float w[6];
#pragma unroll
            for (int q = 0; q < 6; q++) {
              const int n = ((f >> q) & 1u) ? faces[j * 6 + q] : -1;
              w[q] = n >= 0 ? cur[n] : 0.f;
            }
            const float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
            next = bfRound((sum - cr[j]) / fmaxf(diagOf(f & 63u), 1e-12f), nB);
          }
          cur[j] = next;
        }
        __syncthreads();
      }
    }
    for (int it = 0; !RB && it < iterations; it++) {
      if (own < nt) {
        float next = 0.f;
        if (!(ownFlags & SOLIDF)) {
          float w[6];
#pragma unroll
          for (int k = 0; k < 6; k++) w[k] = ownNbr[k] >= 0 ? cur[ownNbr[k]] : 0.f;
          const float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
          next = mixf(cur[own], (sum - ownRhs) / ownDiag, 0.8f);
        }
        nxt[own] = next;
      }
      for (int j = own + blockDim.x; j < nt; j += blockDim.x) {
        const uint32_t f = fb[j];
        float next = 0.f;
        if (!(f & SOLIDF)) {
          float w[6];
#pragma unroll
          for (int k = 0; k < 6; k++) {
            const int n = ((f >> k) & 1u) ? faces[j * 6 + k] : -1;
            w[k] = n >= 0 ? cur[n] : 0.f;
          }
          float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
          float cand = (sum - cr[j]) / fmaxf(diagOf(f & 63u), 1e-12f);
          next = mixf(cur[j], cand, 0.8f);
        }
        nxt[j] = next;
      }
      __syncthreads();
      float* tmp = cur;
      cur = nxt;
      nxt = tmp;
    }
    for (int j = threadIdx.x; j < nt; j += blockDim.x) stBf(A.cfirst, P.liveTiles[j], cur[j], nB);
    __syncthreads();
    // The bottom's stored result at the bottom cell (tile) (dx,dy,dz) from live tile j (slot t):
    // from shared memory as its storage rounds it, from global memory for a tile not live.
    auto bottomNear = [&](int j, int t, int dx, int dy, int dz) {
      const int k = nbrIndex(dx, dy, dz), pos = nb27[j * 27 + k];
      if (pos >= 0) return bfRound(cur[pos], nB);
      if (pos == -1) return 0.f;
      return ldBf(A.cfirst, __ldg(&P.tileNbr[t * 27 + k]), nB);
    };
    // prolongCell at level L from the bottom's stored result, pa -> pb.
    for (int c = threadIdx.x; c < n4; c += blockDim.x) {
      const int t = P.liveTiles[c >> 3], o = c & 7;
      const uint8_t f = fl[c];
      float out = 0.f;
      if ((f & UNKNOWN) && !(f & FP_STORED_SOLID)) {
        int4 rec = __ldg(&P.tileRec[t]);
        Home H = enterTile(P, t, rec);
        int px = rec.x * 2 + (o & 1), py = rec.y * 2 + ((o >> 1) & 1), pz = rec.z * 2 + (o >> 2);
        float qx = ((float)px + 0.5f) * 0.5f - 0.5f, qy = ((float)py + 0.5f) * 0.5f - 0.5f,
              qz = ((float)pz + 0.5f) * 0.5f - 0.5f;
        int ix = (int)floorf(qx), iy = (int)floorf(qy), iz = (int)floorf(qz);
        float fx = qx - floorf(qx), fy = qy - floorf(qy), fz = qz - floorf(qz);
        bool fast = P.colliderCount == 0 && (!P.ground || iy >= 0);
        const int groundY = P.ground ? 0 : -0x7fffffff;
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
          // The ghost's cell (coarseValue mirrors the ground), next to this tile: no solid cell
          // there, so the ghost and the plain sample are both its value.
          const int ox = ix + dx - rec.x, oy = max(iy + dy, groundY) - rec.y, oz = iz + dz - rec.z;
          const bool near = ox >= -1 && ox <= 1 && oy >= -1 && oy <= 1 && oz >= -1 && oz <= 1;
          v[k] = (!anySolid && near) ? bottomNear(c >> 3, t, ox, oy, oz)
                 : fast              ? readAt(P, H, A.cfirst, ix + dx, iy + dy, iz + dz, BL)
                                     : coarseValue(P, H, A.cfirst, BL, ix + dx, iy + dy, iz + dz);
        }
        float corr = mixf(mixf(mixf(v[0], v[1], fx), mixf(v[2], v[3], fx), fy),
                          mixf(mixf(v[4], v[5], fx), mixf(v[6], v[7], fx), fy), fz);
        out = bfRound(pa[c] + corr, nL);
      }
      (RB ? pa : pb)[c] = out;  // a cell reads only its own
    }
    __syncthreads();
    if constexpr (RB) {
      for (int k = 0; k < post * 2; k++) half(1 - (k & 1));
    } else {
      relax(pb, pa);
      relax(pa, pb);
      relax(pb, pa);
    }
    for (int c = threadIdx.x; c < n4; c += blockDim.x) stBf(A.pout, (long)P.liveTiles[c >> 3] * 8 + (c & 7), pa[c], nL);
    __syncthreads();
  }
  waitForPrevious();
}

// The finest level's cells of a brick, for the kernels below: whether one is an unknown (activeCell) and the
// sum of its open neighbours (stencilSum), from the brick's neighbour slots. A general lookup a neighbour
// and a cell was most of their time: on 2.3k bricks 38 us a conjugate-gradient direction, now 18, and on 1k
// 19 us a residual, now 10.
struct FineBrick {
  const int* nslot;
  uint32_t low;  // bit k: the neighbour at minus one on the axes of k's bits computes, or is below the ground
  int N, sh;
  FP_DEV bool unknown(int c) const {
    if (low == 0xffu) return true;
    const int m = (1 << sh) - 1;
    uint32_t sub = 1u;  // the octants whose axes are all on a low face here
    if ((c & m) == 0) sub |= sub << 1;
    if (((c >> sh) & m) == 0) sub |= sub << 2;
    if ((c >> (2 * sh)) == 0) sub |= sub << 4;
    return (~low & sub) == 0u;
  }
  FP_DEV float sum(const float* p, int c, uint32_t f) const {
    const int m = (1 << sh) - 1, x = c & m, y = (c >> sh) & m, z = c >> (2 * sh);
    const int sy = 1 << sh, sz = 1 << (2 * sh);
    auto at = [&](bool open, bool edge, int n, int step, int back) {
      if (!open) return 0.f;
      const long s = nslot[edge ? n : 13];
      return s < 0 ? 0.f : p[s * N + (edge ? c - back : c + step)];
    };
    const float v0 = at(f & 1u, x == m, nbrIndex(1, 0, 0), 1, m), v1 = at(f & 2u, x == 0, nbrIndex(-1, 0, 0), -1, -m);
    const float v2 = at(f & 4u, y == m, nbrIndex(0, 1, 0), sy, m * sy), v3 = at(f & 8u, y == 0, nbrIndex(0, -1, 0), -sy, -m * sy);
    const float v4 = at(f & 16u, z == m, nbrIndex(0, 0, 1), sz, m * sz), v5 = at(f & 32u, z == 0, nbrIndex(0, 0, -1), -sz, -m * sz);
    return (v0 + v1) + (v2 + v3) + (v4 + v5);
  }
};
FP_DEV FineBrick fineBrick(const SimParams& P, const Home& H) {
  FineBrick F{H.nslot, 0u, P.N, P.shift};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dx = -(k & 1), dy = -((k >> 1) & 1), dz = -(k >> 2);
    if ((P.ground && H.by + dy < 0) || H.nslot[nbrIndex(dx, dy, dz)] >= 0) F.low |= 1u << k;
  }
  return F;
}

// The finest level's residual rhs - (sum - diag p) over its unknowns, as restrictCell forms
// it, squared and summed in FP64 per simulation.
__global__ void __launch_bounds__(256) k_residual(FpBatch bt, int pSel, int cycle) {
  __shared__ int nslot[27];
  __shared__ double scratch[32];
  const uint32_t total = workTotal(bt, FP_WORK_ACTIVE);
  FpSolver* sum = nullptr;  // the simulation that the sums belong to
  double r2 = 0.0, b2 = 0.0, n = 0.0;
  auto flush = [&]() {
    if (!sum) return;
    r2 = blockSum(r2, scratch);
    if (cycle == 0) {
      b2 = blockSum(b2, scratch);
      n = blockSum(n, scratch);
    }
    if (threadIdx.x == 0) {
      atomicAdd(&sum->res2[cycle], r2);
      if (cycle == 0) {
        atomicAdd(&sum->rhs2, b2);
        atomicAdd(&sum->unknowns, n);
      }
    }
    r2 = b2 = n = 0.0;
  };
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t i;
    const SimParams& P = *workSim(bt, FP_WORK_ACTIVE, item, i).vview;
    if (cycle > 0 && P.solver->converged) continue;  // the same for the whole CTA
    if (!homeOk(P, P.active[i])) continue;  // the bounds-checked build only
    if (sum != P.solver) {
      flush();
      sum = P.solver;
    }
    __syncthreads();  // the previous brick's neighbours have been read
    const Home H = enterBrick(P, P.active[i], nslot);
    const FineBrick F = fineBrick(P, H);
    const float* p = P.p0[pSel];
    const long slot = nslot[13];
    for (int c = threadIdx.x; c < P.N; c += blockDim.x) {
      const long a = slot * P.N + c;
      const uint32_t f = expandFlags(P.topo[0][a]);
      if ((f & SOLIDF) || !F.unknown(c)) continue;
      const float rhs = P.div[a];
      const float r = rhs - (F.sum(p, c, f) - diagOf(f) * p[a]);
      r2 += (double)r * (double)r;
      b2 += (double)rhs * (double)rhs;
      n += 1.0;
    }
  }
  flush();
}

// The red-black bottom (no reference counterpart): `sweeps` red-black Gauss-Seidel sweeps of
// the bottom level (one cell a tile) in place, every sweep the even tiles (x + y + z) then the
// odd ones, in one CTA per simulation. Same cell arithmetic as relaxCell's red-black branch;
// each value is rounded as the level's storage rounds it. With S.pin -1 the level starts from
// zero. Shared memory by live tile when 24 bytes a tile fit, else in place in global memory.
__global__ void __launch_bounds__(1024) k_bottom_rb(FpBatch bt, MgSel Sl, int sweeps, int smemBytes) {
  extern __shared__ float bottomSmem[];
  const int nbIndex[6] = {nbrIndex(1, 0, 0), nbrIndex(-1, 0, 0), nbrIndex(0, 1, 0),
                          nbrIndex(0, -1, 0), nbrIndex(0, 0, 1), nbrIndex(0, 0, -1)};
  int sims = batchCount(bt);
  for (int sim = blockIdx.x; sim < sims; sim += gridDim.x) {
    const SimParams& P = *bt.sims[sim].vview;
    const Args A = resolve(P, Sl);
    if (A.skip) continue;  // the same for the whole CTA
    const int level = A.level, L = P.liveCount;
    const bool nB = A.poutN;
    auto flagOf = [&](int t) -> uint32_t {  // t is live
      int4 rec = __ldg(&P.tileRec[t]);
      Home H = enterTile(P, t, rec);
      uint32_t f = activeCell(P, H, rec.x, rec.y, rec.z, level) ? expandFlags(P.topo[level][t]) : SOLIDF;
      return f | (((rec.x + rec.y + rec.z) & 1) ? ODD : 0u);
    };
    if ((long)L * 24 <= (long)smemBytes) {
      float* cur = bottomSmem;
      float* rhs = cur + L;
      uint32_t* flags = reinterpret_cast<uint32_t*>(rhs + L);
      int16_t* nb = reinterpret_cast<int16_t*>(flags + L);  // 6 a tile
      for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const int t = P.liveTiles[j];
        const uint32_t f = flagOf(t);
        flags[j] = f;
        rhs[j] = ldBf(A.rhs, t, A.rhsN);
        for (int k = 0; k < 6; k++) {
          int n = ((f >> k) & 1u) ? checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[t * 27 + nbIndex[k]])) : -1;
          nb[j * 6 + k] = (int16_t)(n >= 0 ? P.tileIndex[n] : -1);
        }
        cur[j] = (A.pin && !(f & SOLIDF)) ? ldBf(A.pin, t, A.pinN) : 0.f;
      }
      __syncthreads();
      for (int it = 0; it < sweeps; it++)
        for (int colour = 0; colour < 2; colour++) {
          for (int j = threadIdx.x; j < L; j += blockDim.x) {
            const uint32_t f = flags[j];
            if ((int)((f & ODD) != 0) != colour) continue;
            float next = 0.f;
            if (!(f & SOLIDF)) {
              float w[6];
#pragma unroll
              for (int k = 0; k < 6; k++) {
                const int n = nb[j * 6 + k];
                w[k] = n >= 0 ? cur[n] : 0.f;
              }
              float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
              next = bfRound((sum - rhs[j]) / fmaxf(diagOf(f & 63u), 1e-12f), nB);
            }
            cur[j] = next;
          }
          __syncthreads();
        }
      for (int j = threadIdx.x; j < L; j += blockDim.x) stBf(A.pout, P.liveTiles[j], cur[j], nB);
      __syncthreads();
      continue;
    }
    // In place in global memory (A.pout, the level's storage type).
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
      const int t = P.liveTiles[j];
      const uint32_t f = flagOf(t);
      if (!A.pin || (f & SOLIDF)) stBf(A.pout, t, 0.f, nB);
    }
    __syncthreads();
    for (int it = 0; it < sweeps; it++)
      for (int colour = 0; colour < 2; colour++) {
        for (int j = threadIdx.x; j < L; j += blockDim.x) {
          const int t = P.liveTiles[j];
          const uint32_t f = flagOf(t);
          if ((int)((f & ODD) != 0) != colour || (f & SOLIDF)) continue;
          float w[6];
#pragma unroll
          for (int k = 0; k < 6; k++) {
            int n = ((f >> k) & 1u) ? checkTile(P, FP_SITE_TILE_NBR, __ldg(&P.tileNbr[t * 27 + nbIndex[k]])) : -1;
            w[k] = n >= 0 ? ldBf(A.pout, n, nB) : 0.f;
          }
          float sum = (w[0] + w[1]) + (w[2] + w[3]) + (w[4] + w[5]);
          stBf(A.pout, t, (sum - ldBf(A.rhs, t, A.rhsN)) / fmaxf(diagOf(f & 63u), 1e-12f), nB);
        }
        __syncthreads();
      }
  }
}

// ---- Flexible conjugate gradients on the finest level (FP_KRYLOV_FCG; no reference
// counterpart). A v = diag v - (sum of the open neighbours), the operator the relaxation
// inverts; the residual s = rhs + A x has the sign restrictCell's residual has. A CTA per
// computing brick, a thread per cell; FP64 sums per CTA and simulation, one double atomic each.
//   begin:     x = p, s = rhs + A p; |s|^2 -> res2[0], |rhs|^2 -> rhs2, unknowns
//   dot:       z.q (the new preconditioned residual against the old A d) -> zq[c]
//   direction: beta = -zq[c] / dq[c-1] (0 at c = 1); d = z + beta d, q = A z + beta q (= A d);
//              d.q -> dq[c], d.s -> ds[c]
//   update:    alpha = -ds[c] / dq[c]; x += alpha d, s += alpha q; |s|^2 -> res2[c]
enum FcgOp { FCG_BEGIN = 0, FCG_DOT = 1, FCG_DIRECTION = 2, FCG_UPDATE = 3 };

template <int OP>
__global__ void __launch_bounds__(256) k_fcg(FpBatch bt, int vSel, int cycle) {
  __shared__ int nslot[27];
  __shared__ double scratch[32];
  const uint32_t total = workTotal(bt, FP_WORK_ACTIVE);
  const bool first = cycle <= 1;
  FpSolver* S = nullptr;  // the simulation that the sums belong to
  double s1 = 0.0, s2 = 0.0, s3 = 0.0;
  float beta = 0.f, alpha = 0.f;
  auto flush = [&]() {
    if (!S) return;
    s1 = blockSum(s1, scratch);
    if (OP == FCG_BEGIN || OP == FCG_DIRECTION) s2 = blockSum(s2, scratch);
    if (OP == FCG_BEGIN) s3 = blockSum(s3, scratch);
    if (threadIdx.x == 0) {
      if (OP == FCG_BEGIN) {
        atomicAdd(&S->res2[0], s1);
        atomicAdd(&S->rhs2, s2);
        atomicAdd(&S->unknowns, s3);
      } else if (OP == FCG_DOT) {
        atomicAdd(&S->zq[cycle], s1);
      } else if (OP == FCG_DIRECTION) {
        atomicAdd(&S->dq[cycle], s1);
        atomicAdd(&S->ds[cycle], s2);
      } else {
        atomicAdd(&S->res2[cycle], s1);
      }
    }
    s1 = s2 = s3 = 0.0;
  };
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t i;
    const SimParams& P = *workSim(bt, FP_WORK_ACTIVE, item, i).vview;
    if (cycle > 0 && P.solver->converged) continue;  // the same for the whole CTA
    if (!homeOk(P, P.active[i])) continue;  // the bounds-checked build only
    if (S != P.solver) {
      flush();
      S = P.solver;
      if (OP == FCG_DIRECTION && !first && S->dq[cycle - 1] != 0.0) beta = (float)(-S->zq[cycle] / S->dq[cycle - 1]);
      else beta = 0.f;
      if (OP == FCG_UPDATE && S->dq[cycle] != 0.0) alpha = (float)(-S->ds[cycle] / S->dq[cycle]);
      else alpha = 0.f;
    }
    __syncthreads();  // the previous brick's neighbours have been read
    const Home H = enterBrick(P, P.active[i], nslot);
    const FineBrick F = fineBrick(P, H);
    const long slot = nslot[13];
    const float* v = vSel >= 0 ? P.p0[vSel] : nullptr;  // BEGIN: p; DOT, DIRECTION: z
    float* x = P.p0[2];
    float* sres = P.kry[0];
    float* d = P.kry[1];
    float* q = P.kry[2];
    for (int c = threadIdx.x; c < P.N; c += blockDim.x) {
      const long a = slot * P.N + c;
      const uint32_t f = expandFlags(P.topo[0][a]);
      const bool unknown = !(f & SOLIDF) && F.unknown(c);
      if (OP == FCG_BEGIN) {
        float p = v[a];
        x[a] = p;
        float r = 0.f;
        if (unknown) {
          float rhs = P.div[a];
          r = rhs - (F.sum(v, c, f) - diagOf(f) * p);
          s1 += (double)r * (double)r;
          s2 += (double)rhs * (double)rhs;
          s3 += 1.0;
        }
        sres[a] = r;
      } else if (OP == FCG_DOT) {
        if (unknown) s1 += (double)v[a] * (double)q[a];
      } else if (OP == FCG_DIRECTION) {
        float dn = 0.f, qn = 0.f;
        if (unknown) {
          float z = v[a];
          float az = diagOf(f) * z - F.sum(v, c, f);
          dn = first ? z : z + beta * d[a];
          qn = first ? az : az + beta * q[a];
          s1 += (double)dn * (double)qn;
          s2 += (double)dn * (double)sres[a];
        }
        d[a] = dn;
        q[a] = qn;
      } else {
        if (unknown) {
          x[a] = x[a] + alpha * d[a];
          float r = sres[a] + alpha * q[a];
          sres[a] = r;
          s1 += (double)r * (double)r;
        }
      }
    }
  }
  flush();
}

// Each simulation's decision after V-cycle `cycle`: converged once the residual's RMS is at
// most the tolerance times the right-hand side's. One CTA.
__global__ void k_converge(FpBatch bt, int cycle) {
  int sims = batchCount(bt);
  for (int sim = threadIdx.x; sim < sims; sim += blockDim.x) {
    const SimParams& P = *bt.sims[sim].vview;
    FpSolver* S = P.solver;
    if (cycle > 0 && S->converged) continue;
    S->cycles = cycle + 1;
    double tol = (double)P.tolerance;
    // Done: the residual met the tolerance, or this simulation's own cycle limit is reached
    // (the launch runs as many cycles as its most demanding simulation).
    if ((tol > 0.0 && S->res2[cycle] <= tol * tol * S->rhs2) || cycle + 1 >= P.vcycles) S->converged = 1;
  }
}

// cellTopology (pressure.wgsl:208-222): solid, or the sides whose neighbours are not solid.
FP_DEV uint8_t cellTopology(const SimParams& P, const Home& H, int px, int py, int pz, int level) {
  // solidAt at the centre of a level's cell, ((x + .5) s h) / h + .25 with s = 2^level field
  // cells a level-0 cell side (solidSpan), floors to field cell x s + s/2 (x itself for s = 1).
  const int span = (1 << level) * P.solidSpan, half = span >> 1;
  auto blocked = [&](int x, int y, int z) { return solidFine(P, H, x * span + half, y * span + half, z * span + half); };
  if (blocked(px, py, pz)) return FP_STORED_SOLID;
  uint8_t flags = 0;
  if (!blocked(px + 1, py, pz)) flags |= 1;
  if (!blocked(px - 1, py, pz)) flags |= 2;
  if (!blocked(px, py + 1, pz)) flags |= 4;
  if (!blocked(px, py - 1, pz)) flags |= 8;
  if (!blocked(px, py, pz + 1)) flags |= 16;
  if (!blocked(px, py, pz - 1)) flags |= 32;
  return flags;
}

// buildBrickTopology (pressure.wgsl:259-278): the brick levels of the slots granted this
// step, or (ALL) of every slotted brick of the simulations whose geometry changed.
template <bool ALL>
__global__ void __launch_bounds__(128) k_topo_bricks(FpBatch bt) {
  __shared__ int nslot[27];
  // Every slotted brick is on the ascending list of computing bricks.
  const int kind = ALL ? FP_WORK_ACTIVE : FP_WORK_FRESH;
  uint32_t total = workTotal(bt, kind);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t i;
    const SimParams& P = *workSim(bt, kind, item, i).vview;
    if ((P.topoAll != 0) != ALL) continue;  // uniform across the CTA
    uint32_t id;
    int slot;
    if (ALL) {
      id = P.active[i];
      if (__ldg(&P.tileRec[id >> 6]).w == 0) continue;
      slot = entryPage(P.entries[id]);
    } else {
      id = P.zeroList[2 * i];
      slot = (int)P.zeroList[2 * i + 1];
    }
    if (slot < 0) continue;
    // The brick's neighbour slots in shared memory: every solid test stays within them.
    if (!homeOk(P, id)) continue;  // the bounds-checked build only
    Home H = enterBrick(P, id, nslot);
    int bx = H.bx, by = H.by, bz = H.bz;
    // A brick whose neighbourhood holds no collider's cell has every side of every cell open at every
    // brick level, but for the ground under its lowest cells: cellTopology would return 63 throughout,
    // or 55 there. (Four cells a store, and the bricks on the ground without asking seven places a
    // cell: every brick of 3.1k anew took 57 us beside the prediction, now 44.)
    bool solidNear = P.ground && by < 0;
    if (!solidNear && P.colliderCount > 0) {
      bool any = false;
      for (int q = threadIdx.x; q < 27 * P.W; q += blockDim.x) {
        int s = nslot[q / P.W];
        if (s >= 0 && P.solids[(size_t)s * P.W + q % P.W] != 0u) any = true;
      }
      solidNear = __syncthreads_or(any) != 0;
    }
    if (!solidNear) {
      const bool onGround = P.ground && by == 0;
      for (int level = 0; level < P.brickLevels; level++) {
        const int s = levelShift(P, level), cells = 1 << (3 * s);  // at least 2^3
        uint32_t* out = reinterpret_cast<uint32_t*>(P.topo[level] + (size_t)slot * cells);
        for (int o = threadIdx.x; o < cells / 4; o += blockDim.x) {
          uint32_t flags = 0x3f3f3f3fu;
          if (onGround) {
            if (s > 1 && ((o >> (s - 2)) & ((1 << s) - 1)) == 0) flags = 0x37373737u;  // a row of 4 cells or more
            if (s == 1) flags = 0x3f3f3737u;                                           // both rows of a layer
          }
          out[o] = flags;
        }
      }
      __syncthreads();
      continue;
    }
    for (int level = 0; level < P.brickLevels; level++) {
      int s = levelShift(P, level), side = 1 << s, cells = side * side * side;
      for (int o = threadIdx.x; o < cells; o += blockDim.x) {
        int lx = o & (side - 1), ly = (o >> s) & (side - 1), lz = o >> (2 * s);
        P.topo[level][(size_t)slot * cells + o] = cellTopology(P, H, bx * side + lx, by * side + ly, bz * side + lz, level);
      }
    }
    __syncthreads();
  }
}

// Each tile slot's mask of computing bricks this step (activeCell at the tile levels,
// pressure.wgsl:100-136, asks whether every brick a cell covers has an entry and computes):
// a CTA of 64 threads per tile, a thread per brick.
__global__ void __launch_bounds__(64) k_tile_masks(FpBatch bt) {
  uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item, local).vview;
    const int t = P.liveTiles[local];
    const size_t id = (size_t)t * 64 + threadIdx.x;
    const bool slotted = __ldg(&P.tileRec[t]).w != 0 && P.entries[id] >= 0;
    bool on = slotted && P.records[id * FP_RECORD_WORDS + 27] != 0;
    uint32_t half = __ballot_sync(0xffffffffu, on);
    if ((threadIdx.x & 31) == 0) reinterpret_cast<uint32_t*>(P.tileMask)[2 * t + (threadIdx.x >> 5)] = half;
    // The first tile level's right-hand side and first iterate at a brick without a slot: the
    // restriction into that level writes only slotted bricks' cells (no other has an unknown
    // child, so restrictCell would write zero there).
    if (!slotted) {
      const int L = P.brickLevels;
      const bool narrow = narrowLevel(P, L);
      stBf(P.lrhs[L], (long)id, 0.f, narrow);
      stBf(P.lp[L][1], (long)id, 0.f, narrow);
    }
  }
}

// buildTileTopology (pressure.wgsl:281-305): every tile's cells at the tile levels.
__global__ void __launch_bounds__(64) k_topo_tiles(FpBatch bt) {
  uint32_t total = workTotal(bt, FP_WORK_TILES);
  for (uint32_t item = blockIdx.x; item < total; item += gridDim.x) {
    uint32_t local;
    const SimParams& P = *workSim(bt, FP_WORK_TILES, item, local).vview;
    if (!P.topoAll) continue;
    int t = P.liveTiles[local];
    int4 rec = __ldg(&P.tileRec[t]);
    if (rec.w == 0) continue;
    Home H = enterTile(P, t, rec);
    for (int level = P.brickLevels; level <= P.bottom; level++) {
      int s = levelShift(P, level), side = 1 << s, cells = side * side * side;
      for (int o = threadIdx.x; o < cells; o += blockDim.x) {
        int lx = o & (side - 1), ly = (o >> s) & (side - 1), lz = o >> (2 * s);
        P.topo[level][(size_t)t * cells + o] =
            cellTopology(P, H, rec.x * side + lx, rec.y * side + ly, rec.z * side + lz, level);
      }
    }
  }
}

}  // namespace

void fp_launch_topology(const FpBatch& bt, bool anyAll, int sms, cudaStream_t st) {
  k_tile_masks<<<sms * 16, 64, 0, st>>>(bt);
  k_topo_bricks<false><<<sms * 4, 128, 0, st>>>(bt);
  if (anyAll) {
    k_topo_bricks<true><<<sms * 4, 128, 0, st>>>(bt);
    k_topo_tiles<<<sms * 8, 64, 0, st>>>(bt);
  }
}

static const int BOTTOM_SMEM = 200 * 1024;
// Resident CTAs per SM of each staged tile-level instantiation, from the occupancy calculator.
template <int OP, int TS>
static int& tileStagedCtas() {
  static int n = 4;
  return n;
}
template <int OP, int TS>
static void configureTileStaged() {
  using K = TileStaged<OP, TS>;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_level_tiles_staged<OP, TS>, 256, K::SMEM) != cudaSuccess) n = 4;
  tileStagedCtas<OP, TS>() = n > 0 ? n : 1;
}
template <int OP, int TS>
static void tileStagedLaunch(const FpBatch& bt, const MgSel& S, int sms, cudaStream_t st) {
  k_level_tiles_staged<OP, TS><<<sms * tileStagedCtas<OP, TS>(), 256, TileStaged<OP, TS>::SMEM, st>>>(bt, S);
}

// The leg kernels: which cells a CTA owns.
enum Owner { BRICK8, BRICK4, PAIRS, TILE4 };
template <int OWNER, int LEG>
static auto legKernel() {
  if constexpr (OWNER == BRICK8) return k_leg_bricks<8, LEG>;
  else if constexpr (OWNER == BRICK4) return k_leg_bricks<4, LEG>;
  else if constexpr (OWNER == PAIRS) return k_leg_pairs<LEG>;
  else return k_leg_tiles<LEG>;
}
// Resident CTAs per SM of each, from the occupancy calculator.
template <int OWNER, int LEG>
static int& legCtas() {
  static int n = 4;
  return n;
}
template <int OWNER, int LEG>
static void configureLeg() {
  using K = Rim<OWNER == BRICK8 || OWNER == PAIRS ? 8 : 4, rimOf(LEG)>;
  static_assert(K::SMEM <= 46 * 1024, "with the static arrays within the limit a kernel needs no attribute for");
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, legKernel<OWNER, LEG>(), K::THREADS, K::SMEM);
  legCtas<OWNER, LEG>() = e == cudaSuccess && n > 0 ? n : 4;
}
template <int OWNER, int LEG>
static void legLaunch(const FpBatch& bt, const MgSel& S, int sms, cudaStream_t st) {
  using K = Rim<OWNER == BRICK8 || OWNER == PAIRS ? 8 : 4, rimOf(LEG)>;
  launchChained(S.overlap, legKernel<OWNER, LEG>(), sms * legCtas<OWNER, LEG>(), K::THREADS, K::SMEM, st, bt, S);
}

// Resident CTAs per SM of each staged instantiation, from the occupancy calculator.
template <int OP, int SB>
static int& stagedCtas() {
  static int n = 4;
  return n;
}
template <int OP, int SB>
static void configureStaged() {
  using K = Staged<OP, SB>;
  cudaFuncSetAttribute(k_level_bricks_staged<OP, SB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::SMEM);
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_level_bricks_staged<OP, SB>, 256, K::SMEM) != cudaSuccess)
    n = 4;
  stagedCtas<OP, SB>() = n > 0 ? n : 1;
}
void fp_mg_configure(int B) {
  (void)B;
  configureStaged<RELAX, 32>();
  configureStaged<RELAX, 16>();
  configureStaged<RELAX, 8>();
  configureStaged<RELAX, 4>();
  configureStaged<RELAX, 2>();
  configureStaged<RESTRICT, 32>();
  configureStaged<RESTRICT, 16>();
  configureStaged<RESTRICT, 8>();
  configureStaged<RESTRICT, 4>();
  configureStaged<RESTRICT, 2>();
  configureStaged<PROLONG, 16>();
  configureStaged<PROLONG, 8>();
  configureStaged<PROLONG, 4>();
  configureStaged<PROLONG, 2>();
  configureStaged<PROLONG, 1>();
  configureLeg<BRICK8, REST>();
  configureLeg<BRICK8, DOWN>();
  configureLeg<BRICK8, UP>();
  configureLeg<BRICK8, PUP>();
  configureLeg<BRICK4, REST>();
  configureLeg<BRICK4, DOWN>();
  configureLeg<BRICK4, UP>();
  configureLeg<BRICK4, PUP>();
  configureLeg<PAIRS, DOWN>();
  configureLeg<PAIRS, PUP>();
  configureLeg<TILE4, DOWN>();
  configureLeg<TILE4, PUP>();
  configureLeg<BRICK8, RB>();
  configureLeg<BRICK4, RB>();
  configureLeg<PAIRS, RB>();
  configureLeg<TILE4, RB>();
  configureTileStaged<RESTRICT, 4>();
  configureTileStaged<PROLONG, 2>();
  cudaFuncSetAttribute(k_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, BOTTOM_SMEM);
  cudaFuncSetAttribute(k_bottom_rb, cudaFuncAttributeMaxDynamicSharedMemorySize, BOTTOM_SMEM);
  cudaFuncSetAttribute(k_coarse<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, COARSE_SMEM);
  cudaFuncSetAttribute(k_coarse<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, COARSE_SMEM);
}

template <int OP, int SB>
static void stagedLaunch(const FpBatch& bt, const MgSel& S, int sms, cudaStream_t st) {
  k_level_bricks_staged<OP, SB><<<sms * stagedCtas<OP, SB>(), 256, Staged<OP, SB>::SMEM, st>>>(bt, S);
}

// The staged level's cells per brick side for an operation whose output level is `level`,
// in bricks of B velocity cells a side (1: the first tile level).
static int log2i(int v) {
  int s = 0;
  while ((1 << s) < v) s++;
  return s;
}
template <int OP>
static int stagedSide(int level, int B) {
  int bl = log2i(B);
  int stage = OP == PROLONG ? level + 1 : (OP == RESTRICT ? level - 1 : level);
  return stage < bl ? 1 << (bl - stage) : 1;
}

template <int OP>
static void levelLaunch(const FpBatch& bt, const MgSel& S, bool tiles, int B, int sms, cudaStream_t st) {
  if constexpr (OP == RESTRICT) {
    // Into the first tile level: a brick's cell there restricts the brick's own 2^3 cells, staged
    // per brick like the brick levels. Cells of bricks without a slot have no unknown child and
    // stay zero (k_tile_masks clears them each step).
    if (tiles && S.level == log2i(B)) {
      stagedLaunch<OP, 2>(bt, S, sms, st);
      return;
    }
  }
  if (tiles) {
    // The tile levels hold 4^3, 2^3 and one cell a tile. Operations that read or write the first
    // (a cell a brick) are staged per tile; its sweeps are legs (fp_legs_fused).
    const int below = S.level - log2i(B);
    if (OP == RESTRICT && below == 1) {
      tileStagedLaunch<RESTRICT, 4>(bt, S, sms, st);
      return;
    }
    if (OP == PROLONG && below == 0) {
      tileStagedLaunch<PROLONG, 2>(bt, S, sms, st);
      return;
    }
    if (below == 1)
      k_level_tiles<OP, 8><<<sms * 16, 64, 0, st>>>(bt, S);
    else
      k_level_tiles<OP, 1><<<sms * 16, 64, 0, st>>>(bt, S);
    return;
  }
  // Relaxation stages sides 32..2, restriction its fine sides 32..4, prolongation 16..1.
  const int sb = stagedSide<OP>(S.level, B);
  if constexpr (OP == RELAX) {
    if (sb == 32) stagedLaunch<OP, 32>(bt, S, sms, st);
    else if (sb == 16) stagedLaunch<OP, 16>(bt, S, sms, st);
    else if (sb == 8) stagedLaunch<OP, 8>(bt, S, sms, st);
    else if (sb == 4) stagedLaunch<OP, 4>(bt, S, sms, st);
    else stagedLaunch<OP, 2>(bt, S, sms, st);
  } else if constexpr (OP == RESTRICT) {
    if (sb == 32) stagedLaunch<OP, 32>(bt, S, sms, st);
    else if (sb == 16) stagedLaunch<OP, 16>(bt, S, sms, st);
    else if (sb == 8) stagedLaunch<OP, 8>(bt, S, sms, st);
    else if (sb == 4) stagedLaunch<OP, 4>(bt, S, sms, st);
    else stagedLaunch<OP, 2>(bt, S, sms, st);
  } else {
    if (sb == 16) stagedLaunch<OP, 16>(bt, S, sms, st);
    else if (sb == 8) stagedLaunch<OP, 8>(bt, S, sms, st);
    else if (sb == 4) stagedLaunch<OP, 4>(bt, S, sms, st);
    else if (sb == 2) stagedLaunch<OP, 2>(bt, S, sms, st);
    else stagedLaunch<OP, 1>(bt, S, sms, st);
  }
}
void fp_launch_relax(const FpBatch& bt, const MgSel& S, bool tiles, int B, int sms, cudaStream_t st) {
  levelLaunch<RELAX>(bt, S, tiles, B, sms, st);
}
// The levels whose legs are one launch: brick levels of 8^3, 4^3 and 2^3 cells a brick, and the first
// tile level. (At 16^3 and 32^3 a box does not fit several to an SM, and a step is no longer mostly
// latency; the levels below are k_coarse's.)
bool fp_legs_fused(int level, int B) {
  const int bl = log2i(B), side = level < bl ? B >> level : 0;
  return side == 8 || side == 4 || (side == 2 && level > 0) || level == bl;
}
bool fp_leg_per_brick(int level, int B) { return level < log2i(B) && (B >> level) >= 4; }
template <int LEG>
static void legsLaunch(const FpBatch& bt, const MgSel& S, int B, int sms, cudaStream_t st) {
  const int side = S.level < log2i(B) ? B >> S.level : 0;
  if (side == 8) {
    legLaunch<BRICK8, LEG>(bt, S, sms, st);
  } else if (side == 4) {
    legLaunch<BRICK4, LEG>(bt, S, sms, st);
  } else if constexpr (LEG == DOWN || LEG == PUP || LEG == RB) {
    if (side == 2)
      legLaunch<PAIRS, LEG>(bt, S, sms, st);
    else
      legLaunch<TILE4, LEG>(bt, S, sms, st);
  }
}
void fp_launch_leg_down(const FpBatch& bt, const MgSel& S, int B, int sms, cudaStream_t st) {
  if (S.level == 0)
    legsLaunch<REST>(bt, S, B, sms, st);
  else
    legsLaunch<DOWN>(bt, S, B, sms, st);
}
void fp_launch_leg_up(const FpBatch& bt, const MgSel& S, int B, int sms, cudaStream_t st) {
  if (S.coarse < 0)
    legsLaunch<UP>(bt, S, B, sms, st);
  else
    legsLaunch<PUP>(bt, S, B, sms, st);
}
void fp_launch_leg_rb(const FpBatch& bt, const MgSel& S, int B, int sms, cudaStream_t st) {
  legsLaunch<RB>(bt, S, B, sms, st);
}
void fp_launch_restrict(const FpBatch& bt, const MgSel& S, bool tiles, int B, int sms, cudaStream_t st) {
  levelLaunch<RESTRICT>(bt, S, tiles, B, sms, st);
}
void fp_launch_prolong(const FpBatch& bt, const MgSel& S, bool tiles, int B, int sms, cudaStream_t st) {
  levelLaunch<PROLONG>(bt, S, tiles, B, sms, st);
}
void fp_launch_bottom(const FpBatch& bt, const MgSel& S, int iterations, int sms, cudaStream_t st) {
  k_bottom<<<sms, 1024, BOTTOM_SMEM, st>>>(bt, S, iterations, BOTTOM_SMEM);
}
bool fp_coarse_fits(int liveTiles) { return (long)liveTiles * COARSE_SLOT_BYTES <= COARSE_SMEM; }
// `small`: every simulation has at most COARSE_SMALL live tiles; a CTA a simulation of up to `sims`.
// Fewer warps meet at a barrier sooner, and little shared memory leaves the neighbours' CTAs room. It
// holds a few more, so that a simulation that grows past the line steps on until the other form is there.
constexpr int COARSE_SMALL = 64, COARSE_SMALL_ROOM = 80;
bool fp_coarse_small(int liveTiles) { return liveTiles <= COARSE_SMALL; }
bool fp_coarse_small_holds(int liveTiles) { return liveTiles <= COARSE_SMALL_ROOM; }
void fp_launch_coarse(const FpBatch& bt, const MgSel& S, int iterations, bool small, int sims, int sms, cudaStream_t st) {
  const int smem = small ? COARSE_SMALL_ROOM * COARSE_SLOT_BYTES : COARSE_SMEM;
  launchChained(S.overlap, k_coarse<false>, sims < sms ? sims : sms, small ? 256 : 1024, (size_t)smem, st, bt, S, iterations, smem, 0, 0);
}
void fp_launch_coarse_rb(const FpBatch& bt, const MgSel& S, int pre, int bottom, int post, bool small, int sims, int sms, cudaStream_t st) {
  const int smem = small ? COARSE_SMALL_ROOM * COARSE_SLOT_BYTES : COARSE_SMEM;
  k_coarse<true><<<sims < sms ? sims : sms, small ? 256 : 1024, smem, st>>>(bt, S, bottom, smem, pre, post);
}

void fp_launch_residual(const FpBatch& bt, int pSel, int cycle, int sms, cudaStream_t st) {
  k_residual<<<sms * 4, 256, 0, st>>>(bt, pSel, cycle);
  k_converge<<<1, 256, 0, st>>>(bt, cycle);
}

void fp_launch_bottom_rb(const FpBatch& bt, const MgSel& S, int sweeps, int sms, cudaStream_t st) {
  k_bottom_rb<<<sms, 1024, BOTTOM_SMEM, st>>>(bt, S, sweeps, BOTTOM_SMEM);
}

void fp_launch_fcg_begin(const FpBatch& bt, int pSel, int sms, cudaStream_t st) {
  k_fcg<FCG_BEGIN><<<sms * 4, 256, 0, st>>>(bt, pSel, 0);
  k_converge<<<1, 256, 0, st>>>(bt, 0);
}
int fp_fcg_iterate_launches(int cycle) { return cycle > 1 ? 4 : 3; }
void fp_launch_fcg_iterate(const FpBatch& bt, int zSel, int cycle, int sms, cudaStream_t st) {
  if (cycle > 1) k_fcg<FCG_DOT><<<sms * 4, 256, 0, st>>>(bt, zSel, cycle);
  k_fcg<FCG_DIRECTION><<<sms * 4, 256, 0, st>>>(bt, zSel, cycle);
  k_fcg<FCG_UPDATE><<<sms * 4, 256, 0, st>>>(bt, -1, cycle);
  k_converge<<<1, 256, 0, st>>>(bt, cycle);
}
