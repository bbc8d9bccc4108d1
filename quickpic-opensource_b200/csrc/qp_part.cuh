// qp_part.cuh -- tile-binned plasma particles and their kernels.
#pragma once

#include "qp_common.cuh"

namespace qp {

constexpr int TILE = 16;  // cells per tile side (part2d_class.f03:99, mx = my = 16)
constexpr int TN = TILE + 1;  // nodes per tile side
constexpr int NCOMP = 8;  // x, y, px, py, pz, p6, p7, q  (ppart(1..8))

// Structure-of-arrays particle buffer.
struct PartBuf {
  float* c[NCOMP];
  int* count;  // per tile
  int cap;     // slots per tile
};

// Movers in flight to their destination tile (filled by the push, drained by
// the insert kernel).
struct Inbox {
  float* c[NCOMP];
  unsigned long long* key;  // cell << 48 | source tile << 24 | source slot: deterministic order
  int* count;     // per destination tile
  int cap;        // slots per tile
};

struct TileGeom {
  int nx, ny, mx1, myp1, ntiles;
  int rp;
};

// field planes a particle kernel gathers from (real space): node-major
// (fb, ff; the fused step) or, with fb null, one plane per component
struct GatherPlanes {
  const float4* fb;  // (psit, bx, by, bz)
  const float4* ff;  // (fx, fy, psi, unused)
  const float* fx;   // fxy(1)
  const float* fy;   // fxy(2)
  const float* bx;   // bxyz(1)
  const float* by;   // bxyz(2)
  const float* bz;   // bxyz(3)
  const float* psit; // psit
  int combine;       // 1: the push uses -fxy + (by, -bx), the final slice force
  int ext;           // amjdp only: form p6, p7 from psi first (extpsi); node-major fields
  int pass;          // amjdp only: predictor-corrector pass (pass_skipped), 0 = none
  int hold;          // amjdp only: 1 = the next grid starts at this one's end
  float* zero_q;     // push only, optional: clear the charge-plane nodes this tile
                     // owns (k_insert then deposits the next slice's charge)
  // push with combine only, optional: the slice's fields go to these planes --
  // fxy dex and psit to be, bxy dex and bz to bb -- at plane `cursor` of stacks
  // of store_planes (0: at the pointers themselves)
  float* be[3];
  float* bb[3];
  long long store_stride;
  int store_planes;
};

// places the static scratch of qp_pmove_static on the current device (qp_noalloc.cu)
int pmove_static_reserve();
void launch_deposit_rho(const PartBuf& P, const TileGeom& tg, float* q, const DevStatus* st,
                        cudaStream_t s);
void launch_extpsi(const PartBuf& P, const TileGeom& tg, const float* psi, float qbm, float dex,
                   const DevStatus* st, cudaStream_t s);
void launch_amjdp(const PartBuf& P, const TileGeom& tg, const GatherPlanes& f, float* const* acc,
                  float qbm, float dt, float dex, float scale, const DevStatus* st,
                  cudaStream_t s);
// the same into node-major densities node[y][x][8] (cu x/y/z, dcu x/y, amu
// xx/yy/xy), from node-major fields; cz (optional) also takes the z current
void launch_amjdp_node(const PartBuf& P, const TileGeom& tg, const GatherPlanes& f, float* node,
                       float* cz, float qbm, float dt, float dex, float scale,
                       const DevStatus* st, cudaStream_t s);
// mode 0: push in place (partpush); 1: push A -> B with re-binning (push + pmove);
// 2: re-bin only (pmove) A -> B
void launch_push(int mode, const PartBuf& A, const PartBuf& B, const Inbox& ib,
                 const TileGeom& tg, const GatherPlanes& f, float qbm, float dt, float dex,
                 DevStatus* st, cudaStream_t s);
// A = the particles of P0 (rest of A's slots zero) with charge q P0's times qm
void launch_renew(const PartBuf& P0, const PartBuf& A, int ntiles, float qm, cudaStream_t s);
// deposit_q (optional): after the re-bin, deposit the charge of every
// particle of the tile into deposit_q (zero on entry), as k_deposit_rho does;
// hold = 1: the next grid starts at this one's end
void launch_insert(const PartBuf& B, const Inbox& ib, const TileGeom& tg, DevStatus* st,
                   cudaStream_t s, float* deposit_q = nullptr, int hold = 0);

}  // namespace qp
