// qp_part.cu -- plasma particle kernels on tile-binned structure-of-arrays.
//
// One CTA owns one 16 x 16 cell tile (the reference's tile, part2d_class.f03:99)
// and stages the 17 x 17 field nodes it interpolates from in shared memory.
// The particles of a tile are kept in cell order (k_push), so the deposits sum
// runs of same-cell particles in registers and add each run's corner sums to
// the zeroed global planes with L2 reductions (red.global.add.f32, native for
// FP32, where shared-memory float atomics are compare-and-swap loops).  The
// top edge of the top tile row is folded onto row 0 as it is added -- the
// single-rank guard add PPNACGUARD2L (ufield2d_lib.f03:90-97) done in-kernel.
// Per-particle arithmetic follows the reference routines line by line:
//   deposit_rho  PPGPPOST2L         part2d_lib77.f:194-309
//   extpsi       WPGPSIPOST2L_QP    part2d_lib77.f:2207-2284
//   amjdp        PPGRDCJPPOST2L_QP  part2d_lib77.f:311-768
//   push         PPGRBPPUSHF23L_QP  part2d_lib77.f:1066-1408
//   re-binning   PPPORDERF2LA/PPPORDER2LB part2d_lib77.f:1659-2028 (periodic
//                wrap at re-insertion, part2d_lib77.f:1936-1973)
// Every particle's cell is checked against its tile before it indexes shared
// memory or a plane; a particle outside its tile raises a status error instead.
#include "qp_part.cuh"

#include <algorithm>

namespace qp {

namespace {

__device__ __forceinline__ void raise_error(DevStatus* st, int code) {
  if (st) atomicCAS(&st->error, 0, code);
}

__device__ __forceinline__ void tile_origin(const TileGeom& tg, int t, int* noffp, int* moffp) {
  const int ty = t / tg.mx1;
  *noffp = TILE * (t - tg.mx1 * ty);
  *moffp = TILE * ty;
}

// Stage the same 17 x 17 nodes of np planes (np <= NP; all kernels here run
// 256 threads): every thread issues all its loads from L2 before its first
// store to shared memory, so the planes cost one wait instead of one per load.
template <int NP>
__device__ __forceinline__ void stage_planes(float (*s)[TN * TN], const float* const (&pl)[NP],
                                             int np, const TileGeom& tg, int noffp, int moffp) {
  constexpr int PER = (TN * TN + 255) / 256;
  float v[NP][PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + 256 * k;
    const int a = i % TN, b = i / TN;
    const long long o = (long long)(moffp + b) * tg.rp + noffp + a;
#pragma unroll
    for (int p = 0; p < NP; ++p) v[p][k] = (i < TN * TN && p < np) ? pl[p][o] : 0.f;
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + 256 * k;
#pragma unroll
    for (int p = 0; p < NP; ++p)
      if (i < TN * TN && p < np) s[p][i] = v[p][k];
  }
}

// The force fields of a tile's 17 x 17 nodes in shared memory, interleaved so
// that a particle reads a corner with one 16-byte and one 8-byte access:
// consecutive nodes are distinct banks for a warp of cell-ordered particles,
// and the 6 gathers of 4 corners take 8 load instructions instead of 24.
struct FieldTile {
  float4 b[TN * TN];  // psit, bx, by, bz
  float2 f[TN * TN];  // fx, fy
};

// All loads of a thread before its first shared-memory store (one wait for L2).
// psi (optional) is staged beside them.
template <bool NODE>
__device__ __forceinline__ void stage_fields(FieldTile& s, float* spsi, const GatherPlanes& f,
                                             const TileGeom& tg, int noffp, int moffp) {
  constexpr int PER = (TN * TN + 255) / 256;
  float4 vb[PER], vf[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + 256 * k;
    const int a = i % TN, b = i / TN;
    const long long o = (long long)(moffp + b) * tg.rp + noffp + a;
    vb[k] = vf[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < TN * TN) {
      if constexpr (NODE) {
        vb[k] = f.fb[o];
        vf[k] = f.ff[o];
      } else {
        vb[k] = make_float4(f.psit[o], f.bx[o], f.by[o], f.bz[o]);
        vf[k].x = f.fx[o];
        vf[k].y = f.fy[o];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + 256 * k;
    if (i < TN * TN) {
      s.b[i] = vb[k];
      s.f[i] = make_float2(vf[k].x, vf[k].y);
      if (spsi) spsi[i] = vf[k].z;
    }
  }
}

// bilinear interpolation of one component from its 4 corner values, in the
// reference's order of operations
__device__ __forceinline__ float lerp4(float p00, float p01, float p10, float p11, float amx,
                                       float amy, float dxp, float dyp) {
  float d = amx * p00;
  d = amy * (dxp * p01 + d);
  const float ac = amx * p10;
  return d + dyp * (dxp * p11 + ac);
}

struct Gathered {
  float psit, bx, by, bz, fx, fy;
};
__device__ __forceinline__ Gathered gather6(const FieldTile& s, int nn, int mm, float amx,
                                            float amy, float dxp, float dyp) {
  const int o = mm * TN + nn;
  Gathered g;
  {
    const float2 a = s.f[o], b = s.f[o + 1], c = s.f[o + TN], d = s.f[o + TN + 1];
    g.fx = lerp4(a.x, b.x, c.x, d.x, amx, amy, dxp, dyp);
    g.fy = lerp4(a.y, b.y, c.y, d.y, amx, amy, dxp, dyp);
  }
  const float4 a = s.b[o], b = s.b[o + 1], c = s.b[o + TN], d = s.b[o + TN + 1];
  g.psit = lerp4(a.x, b.x, c.x, d.x, amx, amy, dxp, dyp);
  g.bx = lerp4(a.y, b.y, c.y, d.y, amx, amy, dxp, dyp);
  g.by = lerp4(a.z, b.z, c.z, d.z, amx, amy, dxp, dyp);
  g.bz = lerp4(a.w, b.w, c.w, d.w, amx, amy, dxp, dyp);
  return g;
}

// Add a run's 4 corner charges to the global plane q with L2 reductions
// (red.global.add.f32), folding the top edge of the top tile row onto row 0.
__device__ __forceinline__ void deposit_q(float* q, const TileGeom& tg, int noffp, int moffp,
                                          int cell, const float* acc) {
  const int nn = cell % TN, mm = cell / TN;
  const long long o0 = (long long)(moffp + mm) * tg.rp + noffp + nn;
  const int y1 = moffp + mm + 1;
  const long long o2 = (long long)(y1 == tg.ny ? 0 : y1) * tg.rp + noffp + nn;
  atomicAdd(q + o0, acc[0]);
  atomicAdd(q + o0 + 1, acc[1]);
  atomicAdd(q + o2, acc[2]);
  atomicAdd(q + o2 + 1, acc[3]);
}

// Charge deposit with the run scheme of k_amjdp: 4 consecutive particles per
// thread, corner weights of a run of particles in one cell summed in
// registers, then added to q (which must be zero on entry) by deposit_q.
// The n particles of tile t (all the CTA's threads take part).
__device__ __forceinline__ void deposit_tile(const PartBuf& P, const TileGeom& tg, int t, int n,
                                             float* q, DevStatus* st) {
  int noffp, moffp;
  tile_origin(tg, t, &noffp, &moffp);
  const long long base = (long long)t * P.cap;
  for (int k0 = 4 * threadIdx.x; k0 < n; k0 += 4 * blockDim.x) {
    const float4 X = *reinterpret_cast<const float4*>(P.c[0] + base + k0);
    const float4 Y = *reinterpret_cast<const float4*>(P.c[1] + base + k0);
    const float4 QM = *reinterpret_cast<const float4*>(P.c[7] + base + k0);
    const float xs[4] = {X.x, X.y, X.z, X.w}, ys[4] = {Y.x, Y.y, Y.z, Y.w};
    const float qs[4] = {QM.x, QM.y, QM.z, QM.w};
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    int cell = -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (k0 + j < n) {
        const float x = xs[j], y = ys[j], qm = qs[j];
        int nn = (int)x, mm = (int)y;
        const float dxp = qm * (x - (float)nn);
        const float dyp = y - (float)mm;
        nn -= noffp;
        mm -= moffp;
        if (nn < 0 || nn >= TILE || mm < 0 || mm >= TILE) {
          raise_error(st, -3);
          continue;
        }
        const float amx = qm - dxp, amy = 1.f - dyp;
        const float w0 = amx * amy, w1 = dxp * amy, w2 = amx * dyp, w3 = dxp * dyp;
        const int c = mm * TN + nn;
        if (c != cell) {
          if (cell >= 0) deposit_q(q, tg, noffp, moffp, cell, acc);
          cell = c;
          acc[0] = w0;
          acc[1] = w1;
          acc[2] = w2;
          acc[3] = w3;
        } else {
          acc[0] += w0;
          acc[1] += w1;
          acc[2] += w2;
          acc[3] += w3;
        }
      }
    }
    if (cell >= 0) deposit_q(q, tg, noffp, moffp, cell, acc);
  }
}

__global__ void __launch_bounds__(256) k_deposit_rho(PartBuf P, TileGeom tg, float* q,
                                                     DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  const int t = blockIdx.x;
  const int n = P.count[t];
  if (n < 0 || n > P.cap) {  // a count beyond the tile's slots: never read past them
    if (threadIdx.x == 0) raise_error(st, -6);
    return;
  }
  deposit_tile(P, tg, t, n, q, st);
}

__global__ void __launch_bounds__(256) k_extpsi(PartBuf P, TileGeom tg, const float* psi,
                                                float qbm, float dex, DevStatus* st) {
  grid_dep_sync();
  __shared__ float sp[TN * TN];
  if (st && st->error) return;
  const int t = blockIdx.x;
  int noffp, moffp;
  tile_origin(tg, t, &noffp, &moffp);
  {
    const float* const planes[1] = {psi};
    stage_planes<1>(reinterpret_cast<float(*)[TN * TN]>(sp), planes, 1, tg, noffp, moffp);
  }
  __syncthreads();
  const float dx2 = dex * dex;
  const int n = P.count[t];
  if (n < 0 || n > P.cap) {  // a count beyond the tile's slots: never read past them
    if (threadIdx.x == 0) raise_error(st, -6);
    return;
  }
  const long long base = (long long)t * P.cap;
  for (int k0 = 4 * threadIdx.x; k0 < n; k0 += 4 * blockDim.x) {
    const float4 X = *reinterpret_cast<const float4*>(P.c[0] + base + k0);
    const float4 Y = *reinterpret_cast<const float4*>(P.c[1] + base + k0);
    const float4 VX = *reinterpret_cast<const float4*>(P.c[2] + base + k0);
    const float4 VY = *reinterpret_cast<const float4*>(P.c[3] + base + k0);
    float4 P6 = *reinterpret_cast<const float4*>(P.c[5] + base + k0);
    float4 P7 = *reinterpret_cast<const float4*>(P.c[6] + base + k0);
    const float xs[4] = {X.x, X.y, X.z, X.w}, ys[4] = {Y.x, Y.y, Y.z, Y.w};
    const float vxs[4] = {VX.x, VX.y, VX.z, VX.w}, vys[4] = {VY.x, VY.y, VY.z, VY.w};
    float p6[4] = {P6.x, P6.y, P6.z, P6.w}, p7[4] = {P7.x, P7.y, P7.z, P7.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (k0 + j < n) {
        const float x = xs[j], y = ys[j], vx = vxs[j], vy = vys[j];
        int nn = (int)x, mm = (int)y;
        const float dxp = x - (float)nn, dyp = y - (float)mm;
        nn -= noffp;
        mm -= moffp;
        if (nn < 0 || nn >= TILE || mm < 0 || mm >= TILE) {
          raise_error(st, -3);
          continue;
        }
        const float amx = 1.f - dxp, amy = 1.f - dyp;
        const float* s = sp + mm * TN + nn;
        float dx = amx * s[0];
        dx = amy * (dxp * s[1] + dx);
        const float acx = amx * s[TN];
        dx = dx + dyp * (dxp * s[TN + 1] + acx);
        dx = -dx * dx2 * qbm;
        p7[j] = 1.f + dx;
        p6[j] = dx + (dx2 * (vx * vx + vy * vy) - dx * dx - 2.f * dx) / (2.f * (1.f + dx)) + 1.f;
      }
    }
    *reinterpret_cast<float4*>(P.c[5] + base + k0) = make_float4(p6[0], p6[1], p6[2], p6[3]);
    *reinterpret_cast<float4*>(P.c[6] + base + k0) = make_float4(p7[0], p7[1], p7[2], p7[3]);
  }
}

// bilinear gather at (nn, mm) of a 17 x 17 staged plane, in the reference's order
__device__ __forceinline__ float gather(const float* s, int nn, int mm, float amx, float amy,
                                        float dxp, float dyp) {
  const float* p = s + mm * TN + nn;
  float d = amx * p[0];
  d = amy * (dxp * p[1] + d);
  const float ac = amx * p[TN];
  return d + dyp * (dxp * p[TN + 1] + ac);
}

// One particle of PPGRDCJPPOST2L_QP: the half push and the 8 deposited
// quantities (cu x/y/z, dcu x/y, amu xx/yy/xy) and 4 corner weights.
struct AmjOut {
  float v[8];
  float w[4];
  float p6;
};

__device__ __forceinline__ void amjdp_one(const FieldTile& sf, int nn, int mm, float dxp,
                                          float dyp, float vx, float vy, float p6, float p7,
                                          float qm, float qbm, float qtmh, float dti, float dex,
                                          float idex, AmjOut* o) {
  float amx = 1.f - dxp;
  const float amy = 1.f - dyp;
  // __frcp_rn is the correctly rounded 1/x: the same bits as 1.f / x
  const float inv_part_7 = __frcp_rn(p7);
  const float qtmh1 = qtmh * inv_part_7;
  const float qtmh2 = qtmh1 * p6;
  const Gathered g = gather6(sf, nn, mm, amx, amy, dxp, dyp);
  const float dx = g.fx, dy = g.fy;
  float dz = g.psit, ox = g.bx, oy = g.by, oz = g.bz;
  const float ddx = -1.f * qtmh2 * dx + qtmh * oy;
  const float ddy = -1.f * qtmh2 * dy - qtmh * ox;
  const float acx = vx + ddx, acy = vy + ddy;
  const float omzt = qtmh1 * oz;
  const float omt = omzt * omzt;
  const float anorm = 2.f * __frcp_rn(1.f + omt);  // = 2.f / (1.f + omt): 2 x is exact
  const float rot1 = 0.5f * (1.f - omt);
  const float rot2 = omzt;
  float v1 = (rot1 * acx + rot2 * acy) * anorm + ddx;
  float v2 = (rot1 * acy - rot2 * acx) * anorm + ddy;
  const float qm1 = qm * inv_part_7;
  amx = qm1 * amx;
  dxp = qm1 * dxp;
  ox = 0.5f * (v1 + vx);
  oy = 0.5f * (v2 + vy);
  oz = 0.5f * (1.f + dex * dex * (ox * ox + oy * oy)) * inv_part_7 - 0.5f * p7;
  o->p6 = p7 + oz;
  oz = oz * idex;
  vx = (v1 - vx) * dti;
  vy = (v2 - vy) * dti;
  dz = qbm * (dz + (dx * ox + dy * oy) * dex * dex * inv_part_7);
  o->w[0] = amx * amy;
  o->w[1] = dxp * amy;
  o->w[2] = amx * dyp;
  o->w[3] = dxp * dyp;
  v1 = ox * ox * inv_part_7;
  v2 = oy * oy * inv_part_7;
  const float v3 = ox * oy * inv_part_7;
  vx = vx + ox * dz * inv_part_7;
  vy = vy + oy * dz * inv_part_7;
  o->v[0] = ox;
  o->v[1] = oy;
  o->v[2] = oz;
  o->v[3] = vx;
  o->v[4] = vy;
  o->v[5] = v1;
  o->v[6] = v2;
  o->v[7] = v3;
}

// K consecutive floats (a multiple of K from a tile's 16-byte aligned start)
template <int K>
__device__ __forceinline__ void load_k(const float* p, float (&v)[K]) {
  if constexpr (K == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x;
    v[1] = f.y;
    v[2] = f.z;
    v[3] = f.w;
  } else {
    const float2 f = *reinterpret_cast<const float2*>(p);
    v[0] = f.x;
    v[1] = f.y;
  }
}
template <int K>
__device__ __forceinline__ void store_k(float* p, const float (&v)[K]) {
  if constexpr (K == 4)
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// Where amjdp adds its 8 densities: node-major [y][x][8] (node, the fused
// step) or one plane each.  cz (node form only, optional): the z current also
// goes to this plane.
struct Densities {
  float* node;
  float* cz;
  float* pl[8];
};

__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a),
               "f"(b), "f"(c), "f"(d)
               : "memory");
}

// Add the 8 sums v of one corner to node o: fire-and-forget reductions in L2,
// native for FP32, where a shared-memory float atomic is a compare-and-swap
// loop.  A node's 8 densities are one 32-byte sector: two vector reductions
// from one address in place of eight from eight.
template <bool NODE>
__device__ __forceinline__ void add_node(const Densities& d, long long o, const float (&v)[8]) {
  if constexpr (NODE) {
    float* p = d.node + 8 * o;
    red4(p, v[0], v[1], v[2], v[3]);
    red4(p + 4, v[4], v[5], v[6], v[7]);
    if (d.cz) atomicAdd(d.cz + o, v[2]);
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) atomicAdd(d.pl[q] + o, v[q]);
  }
}

// The left corners' nodes of a cell in the two rows; the top edge of the top
// tile row folds onto row 0 (the single-rank guard add, PPNACGUARD2L).
__device__ __forceinline__ void cell_nodes(const TileGeom& tg, int noffp, int moffp, int cell,
                                           long long* o0, long long* o2) {
  const int nn = cell % TN, mm = cell / TN;
  const int y1 = moffp + mm + 1;
  *o0 = (long long)(moffp + mm) * tg.rp + noffp + nn;
  *o2 = (long long)(y1 == tg.ny ? 0 : y1) * tg.rp + noffp + nn;
}

// Add a run's 4 corners x 8 sums to the densities.
template <bool NODE>
__device__ __forceinline__ void deposit_run(const Densities& d, const TileGeom& tg, int noffp,
                                            int moffp, int cell, const float (&acc)[4][8]) {
  long long o0, o2;
  cell_nodes(tg, noffp, moffp, cell, &o0, &o2);
  add_node<NODE>(d, o0, acc[0]);
  add_node<NODE>(d, o0 + 1, acc[1]);
  add_node<NODE>(d, o2, acc[2]);
  add_node<NODE>(d, o2 + 1, acc[3]);
}

// deposit_run for a lane's last run, merged across lanes: the right corners
// of the previous lane's last run are added to this run's left corners when
// take is set, and this run's right corners are left to the next lane when
// give is set.  Every lane of the warp must call it (the shuffles); a lane
// with no run (cell < 0) only passes values on.
template <bool NODE>
__device__ __forceinline__ void deposit_last(const Densities& d, const TileGeom& tg, int noffp,
                                             int moffp, int cell, float (&acc)[4][8], bool take,
                                             bool give) {
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float r1 = __shfl_up_sync(full, acc[1][q], 1);
    const float r3 = __shfl_up_sync(full, acc[3][q], 1);
    if (take) {
      acc[0][q] += r1;
      acc[2][q] += r3;
    }
  }
  if (cell < 0) return;
  long long o0, o2;
  cell_nodes(tg, noffp, moffp, cell, &o0, &o2);
  add_node<NODE>(d, o0, acc[0]);
  add_node<NODE>(d, o2, acc[2]);
  if (!give) {
    add_node<NODE>(d, o0 + 1, acc[1]);
    add_node<NODE>(d, o2 + 1, acc[3]);
  }
}

// The half push and the deposit of 8 densities x 4 corners.  Bound by issue
// (about 380 instructions per particle, 57 % of issue slots at 3 CTAs per SM)
// and by the reductions in L2, not by memory.  Node-major fields and densities:
// 27.0 -> 24.7 us at 512 x 512 with 2 x 2 particles per cell (28 MB: 1.1 TB/s),
// 79.5 -> 73.7 us at 1024 x 1024; without handing right corners to the next
// lane 27.4 us.
// Each thread takes 4 consecutive particles (float4 loads of each component)
// and keeps the deposits of a run of particles in one cell in registers,
// adding them to the global planes when the cell changes (deposit_run).  With
// the particles of a tile stored cell by cell, runs are long and a warp's
// reductions spread over neighbouring nodes.  The per-particle products are
// those of the reference; only the order in which a node's contributions are
// summed differs.  The planes must be zero on entry.
// K = 4 particles per thread and CTA = tile is the form for grids that fill the
// GPU.  Grids of few tiles leave most of it idle and wait for one CTA's serial
// work: there two CTAs share a tile with 2 particles per thread (64 x 64 grid:
// 10.8 -> 9.0 us, 128 x 128: 11.9 -> 10.2).
template <bool NODE, int K>
__global__ void __launch_bounds__(256, 3) k_amjdp(PartBuf P, TileGeom tg, GatherPlanes f,
                                                  const __grid_constant__ Densities den, float qbm,
                                                  float dt, float dex, float scale,
                                                  DevStatus* st) {
  grid_dep_wait();
  // The deposit of the next of several species has nothing to do before its
  // wait, and its early CTAs would crowd some SMs: it is let in at this one's
  // end (with k_insert: two species at 256 x 256, 32 slices 3.35 -> 3.31 ms).
  if (!f.hold) grid_dep_launch();
  __shared__ FieldTile sf;
  __shared__ float spsi[TN * TN];
  if (st && st->error) return;
  if (pass_skipped(st, f.pass)) return;
  const int t = blockIdx.x;
  int noffp, moffp;
  tile_origin(tg, t, &noffp, &moffp);
  const bool ext = NODE && f.ext;
  // the count is read with the field planes, so the two waits overlap
  const int n = P.count[t];
  stage_fields<NODE>(sf, ext ? spsi : nullptr, f, tg, noffp, moffp);
  __syncthreads();
  const float qtmh = 0.5f * qbm * dt;
  const float dti = 1.f / dt;
  const float idex = 1.f / dex;
  const float dx2 = dex * dex;
  if (n < 0 || n > P.cap) {  // a count beyond the tile's slots: never read past them
    if (threadIdx.x == 0) raise_error(st, -6);
    return;
  }
  const long long base = (long long)t * P.cap;
  const int lane = threadIdx.x & 31;
  // the whole warp loops while one of its lanes has particles (the shuffles
  // of the last runs); a lane past the count reads the tile's first slots and
  // neither deposits nor writes them
  const int first = K == 4 ? 4 * threadIdx.x : K * (threadIdx.x + 256 * blockIdx.y);
  for (int k0 = first; k0 - K * lane < n; k0 += 4 * blockDim.x) {
    const bool live = k0 < n;
    const long long kb = base + (live ? k0 : 0);
    float xs[K], ys[K], vxs[K], vys[K], p6s[K], p7s[K], qms[K];
    load_k<K>(P.c[0] + kb, xs);
    load_k<K>(P.c[1] + kb, ys);
    load_k<K>(P.c[2] + kb, vxs);
    load_k<K>(P.c[3] + kb, vys);
    // with ext, p6 and p7 are formed here from psi (k_extpsi) instead of read
#pragma unroll
    for (int j = 0; j < K; ++j) p6s[j] = p7s[j] = 0.f;
    if (!ext) {
      load_k<K>(P.c[5] + kb, p6s);
      load_k<K>(P.c[6] + kb, p7s);
    }
    load_k<K>(P.c[7] + kb, qms);
    float acc[4][8];
    int cell = -1;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (k0 + j < n) {
        int nn = (int)xs[j], mm = (int)ys[j];
        const float dxp = xs[j] - (float)nn, dyp = ys[j] - (float)mm;
        nn -= noffp;
        mm -= moffp;
        if (nn < 0 || nn >= TILE || mm < 0 || mm >= TILE) {
          raise_error(st, -3);
          continue;
        }
        if (ext) {
          // WPGPSIPOST2L_QP for this particle, the same arithmetic as k_extpsi
          float d = gather(spsi, nn, mm, 1.f - dxp, 1.f - dyp, dxp, dyp);
          d = -d * dx2 * qbm;
          p7s[j] = 1.f + d;
          p6s[j] = d + (dx2 * (vxs[j] * vxs[j] + vys[j] * vys[j]) - d * d - 2.f * d) /
                           (2.f * (1.f + d)) +
                   1.f;
        }
        AmjOut o;
        amjdp_one(sf, nn, mm, dxp, dyp, vxs[j], vys[j], p6s[j], p7s[j], qms[j], qbm, qtmh, dti,
                  dex, idex, &o);
        p6s[j] = o.p6;
        // the moments only feed the deposit: the scale goes on the corner
        // weights and the run sums use fused multiply-adds (FP32 roundoff of
        // the sums, like the order of the reductions)
        float ws[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) ws[r] = o.w[r] * scale;
        const int c = mm * TN + nn;
        if (c != cell) {
          if (cell >= 0) deposit_run<NODE>(den, tg, noffp, moffp, cell, acc);
          cell = c;
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[r][q] = o.v[q] * ws[r];
        } else {
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[r][q] = __fmaf_rn(o.v[q], ws[r], acc[r][q]);
        }
      }
    }
    // the last run's right corners go to the next lane when its last run is
    // in the next cell in x (cell + 1 is never a cell at a tile row's end)
    const unsigned full = 0xffffffffu;
    int cprev = __shfl_up_sync(full, cell, 1);
    int cnext = __shfl_down_sync(full, cell, 1);
    if (lane == 0) cprev = -1;
    if (lane == 31) cnext = -1;
    deposit_last<NODE>(den, tg, noffp, moffp, cell, acc, cprev >= 0 && cell == cprev + 1,
                 cell >= 0 && cnext == cell + 1);
    if (live) {
      store_k<K>(P.c[5] + base + k0, p6s);
      if (ext) store_k<K>(P.c[6] + base + k0, p7s);
    }
  }
}

// Push (mode 0, 1) and/or re-bin (mode 1, 2).  Mode 0 writes the pushed
// particles back in place.  In modes 1 and 2 the particles that stay are
// written to B's tile sorted by cell: the tile is taken in chunks of 1024
// slots, the stayers of a chunk are held in shared memory and written out in
// the order of a stable counting sort on their cell, so that the deposits see
// runs of same-cell particles (k_deposit_rho, k_amjdp).  Warp w takes the
// slots w * 128 .. w * 128 + 127 of a chunk, 32 per round, so a particle's
// rank among the earlier same-cell stayers needs only its own warp's running
// counts, and the chunk needs four CTA barriers.  Movers go to the
// destination tile's inbox with a (cell, source tile, source slot) key, which
// the insert kernel sorts, so they too arrive in cell order.
// Bound by issue (550 instructions per particle, 68 % of issue slots; its
// divisions and roots are the reference's IEEE operations): 32 us at 512 x 512
// (1.9 TB/s with the slice's stores, which were a launch of 10.7 us and cost
// 1.3 us here).  A chunk of 1152 slots, which would hold a tile of 1024 and its
// movers, is slower (35 us): five rounds per warp, the last half empty.
constexpr int PUSH_CHUNK = 1024;

template <int MODE>
__global__ void __launch_bounds__(256) k_push(PartBuf A, PartBuf B, Inbox ib, TileGeom tg,
                                              GatherPlanes f, float qbm, float dt, float dex,
                                              DevStatus* st) {
  grid_dep_sync();
  constexpr int CH = MODE != 0 ? PUSH_CHUNK : 1;
  constexpr int NC = MODE != 0 ? 256 : 1;
  constexpr int NR = MODE != 0 ? CH / 256 : 1;  // rounds of 256 slots per chunk
  __shared__ FieldTile sf;
  __shared__ float stg[NCOMP][CH];      // the chunk's stayers, by chunk slot
  __shared__ short perm[CH];            // output order -> chunk slot
  __shared__ unsigned char wcnt[8][NC];  // per warp: its stayers of each cell so far
  __shared__ short woff[8][NC];         // per warp: first output position of each cell
  __shared__ int wtot[8];
  if (st && st->error) return;
  const int t = blockIdx.x;
  int noffp, moffp;
  tile_origin(tg, t, &noffp, &moffp);
  const int n = A.count[t];  // read with the field planes: the waits overlap
  if (f.zero_q) {
    // the tile's 16 x 16 nodes of the charge plane, and on the last tile
    // column / row the rest of the row pitch / the guard row: every node of
    // the plane is cleared by exactly one tile
    const int x1 = (noffp + TILE >= tg.nx) ? tg.rp : noffp + TILE;
    const int y1 = (moffp + TILE >= tg.ny) ? tg.ny + 1 : moffp + TILE;
    const int w = x1 - noffp, h = y1 - moffp;
    for (int i = threadIdx.x; i < w * h; i += blockDim.x)
      f.zero_q[(long long)(moffp + i / w) * tg.rp + noffp + i % w] = 0.f;
  }
  if (MODE != 2) {
    if (f.fb)
      stage_fields<true>(sf, nullptr, f, tg, noffp, moffp);
    else
      stage_fields<false>(sf, nullptr, f, tg, noffp, moffp);
    __syncthreads();
    if (f.combine) {
      long long so = 0;
      if (f.be[0] && f.store_planes) {
        const int cur = st->cursor;
        if (cur < 0 || cur >= f.store_planes) {  // never store outside the 3D arrays
          if (threadIdx.x == 0) raise_error(st, -7);
          return;
        }
        so = cur * f.store_stride;
      }
      // the slice's final force: fxy = -fxy + (bxyz(2), -bxyz(1)), simulation_class.f03:722-724;
      // and the slice's stores (727-735): fxy dex and psit, bxy dex and bz.  The
      // nodes are already here, so the stores cost 6 coalesced 64-byte writes per
      // tile row where a kernel of its own read 6 planes, wrote 10 and was a launch
      const int x1 = noffp + TILE >= tg.nx ? TN : TILE, y1 = moffp + TILE >= tg.ny ? TN : TILE;
      for (int i = threadIdx.x; i < TN * TN; i += blockDim.x) {
        const float4 b = sf.b[i];
        const float2 v = sf.f[i];
        const float fx = -1.f * v.x, fy = -1.f * v.y;
        const float gx = fx + b.z, gy = fy - b.y;
        sf.f[i] = make_float2(gx, gy);
        const int nx = i % TN, ny = i / TN;
        if (f.be[0] && nx < x1 && ny < y1) {  // every node is stored by one tile
          const long long o = so + (long long)(moffp + ny) * tg.rp + noffp + nx;
          f.be[0][o] = gx * dex;
          f.be[1][o] = gy * dex;
          f.be[2][o] = b.x;
          f.bb[0][o] = b.y * dex;
          f.bb[1][o] = b.z * dex;
          f.bb[2][o] = b.w;
        }
      }
    }
  }
  if (MODE != 0)
    for (int i = threadIdx.x; i < 8 * NC; i += blockDim.x) (&wcnt[0][0])[i] = 0;
  __syncthreads();
  const float idex = 1.f / dex;
  const float qtmh = 0.5f * qbm * dt;
  const float anx = (float)tg.nx, any = (float)tg.ny;
  const float edgelx = (float)noffp, edgerx = (float)(noffp + TILE);
  const float edgely = (float)moffp, edgery = (float)(moffp + TILE);
  if (n < 0 || n > A.cap) {  // a count beyond the tile's slots: never read past them
    if (threadIdx.x == 0) raise_error(st, -6);
    return;
  }
  const long long base = (long long)t * A.cap;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  int written = 0;  // stayers written to B so far (the same in every thread)
  for (int c0 = 0; c0 < n; c0 += (MODE != 0 ? CH : (int)blockDim.x)) {
    int cellr[NR];
    // with re-binning the kernel never writes A: its particles are read with
    // read-only loads, and each round's are requested one round ahead, so
    // the wait for L2 overlaps the previous round's push
    float pn[NCOMP];
    {
      const int k = c0 + (MODE != 0 ? warp * (CH / 8) + lane : (int)threadIdx.x);
      if (MODE != 0 && k < n) {
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) pn[c] = __ldg(A.c[c] + base + k);
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int slot = MODE != 0 ? warp * (CH / 8) + r * 32 + lane : threadIdx.x;
      const int k = c0 + slot;
      cellr[r] = -1;
      float pc[NCOMP];
      if (MODE != 0) {
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) pc[c] = pn[c];
        const int kn = k + 32;  // the next round's slot
        if (r + 1 < NR && kn < n) {
#pragma unroll
          for (int c = 0; c < NCOMP; ++c) pn[c] = __ldg(A.c[c] + base + kn);
        }
      }
      if (k >= n) continue;
      if (MODE == 0) {
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) pc[c] = A.c[c][base + k];
      }
      if (MODE != 2) {
        const float x = pc[0], y = pc[1];
        int nn = (int)x, mm = (int)y;
        const float p6 = pc[5], p7 = pc[6];
        const float qtmh1 = qtmh / p7;
        const float qtmh2 = qtmh1 * p6;
        const float dxp = x - (float)nn, dyp = y - (float)mm;
        nn -= noffp;
        mm -= moffp;
        if (nn < 0 || nn >= TILE || mm < 0 || mm >= TILE) {
          raise_error(st, -3);
          nn = 0;
          mm = 0;
        }
        const float amx = 1.f - dxp, amy = 1.f - dyp;
        const Gathered g = gather6(sf, nn, mm, amx, amy, dxp, dyp);
        float dx = g.fx, dy = g.fy, dz = g.psit;
        dz = dz * idex;
        float ox = g.bx, oy = g.by;
        const float oz = g.bz;
        ox = ox * dex;
        oy = oy * dex;
        dx = qtmh2 * dx;
        dy = qtmh2 * dy;
        dz = qtmh2 * dz;
        const float acx = pc[2] + dx, acy = pc[3] + dy, acz = pc[4] + dz;
        const float omxt = qtmh1 * ox, omyt = qtmh1 * oy, omzt = qtmh1 * oz;
        float omt = omxt * omxt + omyt * omyt + omzt * omzt;
        const float anorm = 2.f * __frcp_rn(1.f + omt);  // = 2.f / (1.f + omt)
        omt = 0.5f * (1.f - omt);
        float rot4 = omxt * omyt, rot7 = omxt * omzt, rot8 = omyt * omzt;
        const float rot1 = omt + omxt * omxt, rot5 = omt + omyt * omyt, rot9 = omt + omzt * omzt;
        const float rot2 = omzt + rot4;
        rot4 = -omzt + rot4;
        const float rot3 = -omyt + rot7;
        rot7 = omyt + rot7;
        const float rot6 = omxt + rot8;
        rot8 = -omxt + rot8;
        dx = (rot1 * acx + rot2 * acy + rot3 * acz) * anorm + dx;
        dy = (rot4 * acx + rot5 * acy + rot6 * acz) * anorm + dy;
        dz = (rot7 * acx + rot8 * acy + rot9 * acz) * anorm + dz;
        pc[2] = dx;
        pc[3] = dy;
        pc[4] = dz;
        const float dtc1 = dt / (sqrtf(1.f + (dx * dx + dy * dy + dz * dz) * dex * dex) - dz * dex);
        dx = x + dx * dtc1;
        dy = y + dy * dtc1;
        pc[0] = dx;
        pc[1] = dy;
        // the push's own boundary handling (part2d_lib77.f:1350-1378)
        if (!(dx >= edgerx) && dx < edgelx && dx < 0.f) {
          if (dx + anx >= anx) pc[0] = 0.f;
        }
        if (!(dy >= edgery) && dy < edgely && dy < 0.f) {
          if (dy + any >= any) pc[1] = 0.f;
        }
      }
      if (MODE == 0) {
#pragma unroll
        for (int c = 0; c < 5; ++c) A.c[c][base + k] = pc[c];
        continue;
      }
      // re-insertion wrap of PPPORDER2LB (part2d_lib77.f:1936-1973)
      float xw = pc[0], yw = pc[1];
      if (xw < 0.f) xw = xw + anx;
      if (xw >= anx) xw = xw - anx;
      if (yw < 0.f) yw = yw + any;
      if (yw >= any) yw = yw - any;
      pc[0] = xw;
      pc[1] = yw;
      const int ix = (int)xw, iy = (int)yw;
      int tx = ix / TILE, ty = iy / TILE;
      if (tx < 0 || tx >= tg.mx1 || ty < 0 || ty >= tg.myp1 || !(xw == xw) || !(yw == yw)) {
        raise_error(st, -4);
        tx = 0;
        ty = 0;
      }
      const int dest = tx + tg.mx1 * ty;
      const int cell = (iy & (TILE - 1)) * TILE + (ix & (TILE - 1));
      if (dest == t) {
        cellr[r] = cell;
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) stg[c][slot] = pc[c];
      } else {
        const int islot = atomicAdd(&ib.count[dest], 1);
        if (islot < ib.cap) {
          const long long o = (long long)dest * ib.cap + islot;
#pragma unroll
          for (int c = 0; c < NCOMP; ++c) ib.c[c][o] = pc[c];
          ib.key[o] = ((unsigned long long)cell << 48) | ((unsigned long long)t << 24) |
                      (unsigned long long)(k & 0xffffff);
        } else {
          raise_error(st, QP_OVERFLOW);
          atomicMax(&st->need_inbox, islot + 1);
        }
      }
    }
    if constexpr (MODE != 0) {
      // rank of each stayer among the same-cell stayers of lower slots in its
      // warp: the warp's running count of the cell plus the lower lanes of this
      // round that share the cell (warp-local, so __syncwarp suffices)
      int rank[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int cl = cellr[r];
        const unsigned same = __match_any_sync(0xffffffffu, cl >= 0 ? cl : 256 + lane);
        rank[r] = cl >= 0 ? wcnt[warp][cl] + __popc(same & lt) : 0;
        __syncwarp();
        if (cl >= 0 && lane == __ffs(same) - 1) wcnt[warp][cl] += (unsigned char)__popc(same);
        __syncwarp();
      }
      __syncthreads();
      // thread c: the chunk's stayers of cell c, an exclusive scan over the cells,
      // and the first position of each warp's stayers of cell c
      int nst;
      {
        const int c = threadIdx.x;
        int v = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += wcnt[w][c];
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += u;
        }
        if (lane == 31) wtot[warp] = inc;
        __syncthreads();
        int off = 0;
        nst = 0;
        for (int w = 0; w < 8; ++w) {
          if (w < warp) off += wtot[w];
          nst += wtot[w];
        }
        int pos = off + inc - v;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          woff[w][c] = (short)pos;
          pos += wcnt[w][c];
          wcnt[w][c] = 0;  // ready for the next chunk (read again only after a barrier)
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int cl = cellr[r];
        if (cl >= 0) {
          const int pos = woff[warp][cl] + rank[r];
          if (pos >= 0 && pos < CH)
            perm[pos] = (short)(warp * (CH / 8) + r * 32 + lane);
          else
            raise_error(st, -8);
        }
      }
      __syncthreads();
      // write the chunk's stayers in cell order
      for (int j = threadIdx.x; j < nst; j += blockDim.x) {
        const int slot = perm[j];
        const int pos = written + j;
        if (slot < 0 || slot >= CH) {
          raise_error(st, -8);
        } else if (pos < B.cap) {
          const long long o = (long long)t * B.cap + pos;
#pragma unroll
          for (int c = 0; c < NCOMP; ++c) B.c[c][o] = stg[c][slot];
        } else {
          raise_error(st, QP_OVERFLOW);
          atomicMax(&st->need_cap, pos + 1);
        }
      }
      written += nst;
      __syncthreads();
    }
  }
  if (MODE != 0 && threadIdx.x == 0) B.count[t] = written;
}

// Sorts n (key, index) pairs by key, ascending, with all threads of the CTA:
// bitonic merges whose comparators all point the same way (the first step of a
// merge compares with the mirrored element), so that n may be any number:
// what lies past it would stay there and is not touched.
template <typename I>
__device__ __forceinline__ void sort_pairs(unsigned long long* key, I* idx, int n) {
  int p2 = 1;
  while (p2 < n) p2 <<= 1;
  for (int k = 2; k <= p2; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int o = j == k >> 1 ? i ^ (k - 1) : i ^ j;
        if (o > i && o < n) {
          const unsigned long long a = key[i], b = key[o];
          if (a > b) {
            key[i] = b;
            key[o] = a;
            const I t = idx[i];
            idx[i] = idx[o];
            idx[o] = t;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Insert the movers of tile t after its stayers, sorted by their key so that
// the particle order does not depend on the order in which the atomics of the
// push handed out inbox slots.  One size of shared memory serves any inbox: up
// to one mover per thread is placed by rank, up to INSERT_SORT are sorted in
// shared memory, and more in the inbox itself with the movers' slots of the
// output as the index array (a tile of 8 x 8 particles per cell, 16384 in all,
// takes in 1000 per cell width that its neighbours' plasma moves in a slice).
// At most 32 registers: 8 CTAs per SM hold the 1024 tiles of a 512 x 512 grid in
// one wave (6 left a second one of 136 CTAs).  The shared memory, 10 KB, is what
// a CTA keeps from the kernels of other streams: sized by the inbox (24 KB at
// 2 x 2 particles per cell, 96 KB at 4 x 4) it cost a scan of 64 instances 4 %
// (6.78 against 7.07e9 particle-slices/s with 8 workers).
constexpr int INSERT_SORT = 1024;
__global__ void __launch_bounds__(256, 8) k_insert(PartBuf B, Inbox ib, TileGeom tg, DevStatus* st,
                                                   float* dq, int hold) {
  grid_dep_wait();
  if (!hold) grid_dep_launch();  // as in k_amjdp: the next species' push follows
  __shared__ unsigned long long skey[INSERT_SORT];
  __shared__ short sidx[INSERT_SORT];
  if (st && st->error) return;
  const int t = blockIdx.x;
  int nin = ib.count[t];
  if (nin > ib.cap) {
    raise_error(st, QP_OVERFLOW);
    atomicMax(&st->need_inbox, nin);
    return;
  }
  const int stay = B.count[t];
  if (stay < 0 || stay > B.cap) {
    if (threadIdx.x == 0) raise_error(st, -6);
    return;
  }
  if (stay + nin > B.cap) {
    raise_error(st, QP_OVERFLOW);
    atomicMax(&st->need_cap, stay + nin);
    return;
  }
  const long long ib0 = (long long)t * ib.cap, ob = (long long)t * B.cap + stay;
  if (nin <= (int)blockDim.x) {
    // one mover per thread: its place is the number of smaller keys (the keys
    // differ), found without the sort's barriers (a 512 x 512 step moves 20 to
    // 60 particles into a tile: 21 barriers of a bitonic sort).  The mover's
    // components are on their way meanwhile.
    const int i = threadIdx.x;
    unsigned long long key = 0;
    float v[NCOMP];
    if (i < nin) {
      key = ib.key[ib0 + i];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) v[c] = ib.c[c][ib0 + i];
      skey[i] = key;
    }
    __syncthreads();
    if (i < nin) {
      int rank = 0;
      for (int k = 0; k < nin; ++k) rank += skey[k] < key || (skey[k] == key && k < i) ? 1 : 0;
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) B.c[c][ob + rank] = v[c];
    }
  } else {
    const bool shared = nin <= INSERT_SORT;
    int* gidx = reinterpret_cast<int*>(B.c[0] + ob);
    for (int i = threadIdx.x; i < nin; i += blockDim.x) {
      if (shared) {
        skey[i] = ib.key[ib0 + i];
        sidx[i] = (short)i;
      } else {
        gidx[i] = i;
      }
    }
    __syncthreads();
    if (shared)
      sort_pairs(skey, sidx, nin);
    else
      sort_pairs(ib.key + ib0, gidx, nin);
    for (int i = threadIdx.x; i < nin; i += blockDim.x) {
      // slot i of the output is written below, by the thread that reads it here
      const int si = shared ? sidx[i] : gidx[i];
      if (si < 0 || si >= nin) {  // the sort must map the keys onto filled slots
        raise_error(st, -8);
        continue;
      }
      const long long src = ib0 + si;
      // all loads before the stores, so the mover waits for L2 once
      float v[NCOMP];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) v[c] = ib.c[c][src];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) B.c[c][ob + i] = v[c];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    B.count[t] = stay + nin;
    ib.count[t] = 0;
  }
  // the next slice's charge: every particle of the re-binned tile (the
  // movers were written above; the barrier makes them visible to the CTA)
  if (dq) deposit_tile(B, tg, t, stay + nin, dq, st);
}

// species2d%renew on the device: one read of the pristine particles and one
// write of the live buffer, component blockIdx.y, four slots per thread (in
// place of a fill, a strided copy per component and a scaling pass over q).
// Both capacities are multiples of 4, so a float4 never spans two tiles.
__global__ void __launch_bounds__(256) k_renew(const __grid_constant__ PartBuf P0,
                                               const __grid_constant__ PartBuf A, int ntiles,
                                               float qm) {
  grid_dep_sync();
  const int c = blockIdx.y;
  const int na = A.cap >> 2, np = P0.cap >> 2;
  const long long n4 = (long long)ntiles * na;
  const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long i = i0; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / na;
    const int k = (int)(i - t * na);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < np) v = reinterpret_cast<const float4*>(P0.c[c])[t * np + k];
    if (c == 7) v = make_float4(v.x * qm, v.y * qm, v.z * qm, v.w * qm);
    reinterpret_cast<float4*>(A.c[c])[i] = v;
  }
  if (c == 0)
    for (long long t = i0; t < ntiles; t += (long long)gridDim.x * blockDim.x)
      A.count[t] = P0.count[t];
}

}  // namespace

void launch_insert(const PartBuf& B, const Inbox& ib, const TileGeom& tg, DevStatus* st,
                   cudaStream_t s, float* deposit_q, int hold) {
  launch_pdl(k_insert, tg.ntiles, 256, 0, s, B, ib, tg, st, deposit_q, hold);
}

void launch_renew(const PartBuf& P0, const PartBuf& A, int ntiles, float qm, cudaStream_t s) {
  const long long n4 = (long long)ntiles * (A.cap >> 2);
  const long long blocks = std::max(1LL, std::min((n4 + 255) / 256, 148LL * 8));
  launch_pdl(k_renew, dim3((unsigned)blocks, NCOMP), 256, 0, s, P0, A, ntiles, qm);
}

void launch_deposit_rho(const PartBuf& P, const TileGeom& tg, float* q, const DevStatus* st,
                        cudaStream_t s) {
  launch_pdl(k_deposit_rho, tg.ntiles, 256, 0, s, P, tg, q, const_cast<DevStatus*>(st));
}

void launch_extpsi(const PartBuf& P, const TileGeom& tg, const float* psi, float qbm, float dex,
                   const DevStatus* st, cudaStream_t s) {
  launch_pdl(k_extpsi, tg.ntiles, 256, 0, s, P, tg, psi, qbm, dex, const_cast<DevStatus*>(st));
}

void launch_amjdp(const PartBuf& P, const TileGeom& tg, const GatherPlanes& f, float* const* acc,
                  float qbm, float dt, float dex, float scale, const DevStatus* st,
                  cudaStream_t s) {
  Densities d{};
  for (int i = 0; i < 8; ++i) d.pl[i] = acc[i];
  launch_pdl(k_amjdp<false, 4>, tg.ntiles, 256, 0, s, P, tg, f, d, qbm, dt, dex, scale,
             const_cast<DevStatus*>(st));
}

void launch_amjdp_node(const PartBuf& P, const TileGeom& tg, const GatherPlanes& f, float* node,
                       float* cz, float qbm, float dt, float dex, float scale,
                       const DevStatus* st, cudaStream_t s) {
  Densities d{};
  d.node = node;
  d.cz = cz;
  // two CTAs per tile while they all fit at once, 3 per SM of 148 = 444; past
  // that a second wave costs more than it saves (256 x 256, 512 CTAs at the 4
  // per SM that 64 registers allow: 14.8 us against 14.4).  Shorter runs, so
  // more of a node's sum is formed in L2; its error against float64 is the same
  // (B_perp after 16 slices, 24 seeds: 64 x 64 1.21e-6 +- 0.02 against 1.24 +-
  // 0.02 with one CTA, 128 x 128 1.51 +- 0.04 against 1.52 +- 0.03)
  if (tg.ntiles <= 222)
    launch_pdl(k_amjdp<true, 2>, dim3(tg.ntiles, 2), 256, 0, s, P, tg, f, d, qbm, dt, dex, scale,
               const_cast<DevStatus*>(st));
  else
    launch_pdl(k_amjdp<true, 4>, tg.ntiles, 256, 0, s, P, tg, f, d, qbm, dt, dex, scale,
               const_cast<DevStatus*>(st));
}

void launch_push(int mode, const PartBuf& A, const PartBuf& B, const Inbox& ib,
                 const TileGeom& tg, const GatherPlanes& f, float qbm, float dt, float dex,
                 DevStatus* st, cudaStream_t s) {
  if (mode == 0)
    launch_pdl(k_push<0>, tg.ntiles, 256, 0, s, A, B, ib, tg, f, qbm, dt, dex, st);
  else if (mode == 1)
    launch_pdl(k_push<1>, tg.ntiles, 256, 0, s, A, B, ib, tg, f, qbm, dt, dex, st);
  else
    launch_pdl(k_push<2>, tg.ntiles, 256, 0, s, A, B, ib, tg, f, qbm, dt, dex, st);
}

}  // namespace qp
