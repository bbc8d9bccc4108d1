// qp_fft.cuh -- launch interface of the 2D sine/cosine transform passes.
#pragma once

#include "qp_common.cuh"
#include "qp_solve.cuh"

namespace qp {

struct LineTablesHost {
  char* base = nullptr;
  LineTables t{};
  int logn = 0;
};

int line_tables_build(LineTablesHost* t, int logn);
void line_tables_free(LineTablesHost* t);

constexpr int QP_MAX_JOB = 12;

// One component of an x pass.  xfwd: src/src2 are real planes, dst a k plane;
// xinv: src is a k plane, dst a real plane.  cursor_stride != 0 offsets the
// real-space side by cursor * cursor_stride floats (slice of a 3D array chosen
// by the device slice cursor).
struct XComp {
  const float* src;
  const float* src2;
  float* dst;
  float scale;
  int parity;  // 0 sine, 1 cosine
  long long cursor_stride;
  int cursor_planes;  // planes of that 3D array: a cursor outside them raises an error
  int cursor_next;    // 1: the plane after the cursor (before k_slice_a has moved it on)
};
struct XJob {
  XComp c[QP_MAX_JOB];
  int ncomp;
};

struct YComp {
  float* plane;
  float scale;
  int parity;
};
struct YJob {
  YComp c[QP_MAX_JOB];
  int ncomp;
};

int fft_kernels_init();
size_t xpass_smem(const GridDims& g);
size_t ypass_smem(const GridDims& g);
void launch_xfwd(const XJob& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                 cudaStream_t s);
void launch_xinv(const XJob& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                 cudaStream_t s);
// Inverse x pass of the fused step's node-major fields: group g is
// src [kx][y][4] -> dst [y][x][4] with the x parities par[g]; planar components
// (c[0..ncomp), as launch_xinv) ride along, and the launch clears the zero
// planes.
struct X4Job {
  const float4* src[2];
  float4* dst[2];
  int par[2][4];
  int ngroup;
  XJob x;
  float* zero[16];  // planes that this launch clears
  int nzero;
  int pass;  // predictor-corrector pass of the launch (pass_skipped), 0 = none
  int hold;  // 1: the next grid starts at this one's end
};
void launch_xinv4(const X4Job& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                  cudaStream_t s);
// Forward x pass of the fused step's node-major densities: src [y][x][8] ->
// dst [kx][y][8] with the x parities par, rows y < ny (row ny of both stays
// zero: the deposits fold it onto row 0); planar components ride along.
struct X8Job {
  const float4* src;  // two per node
  float4* dst;
  int par[8];
  XJob x;
  int pass;  // as X4Job
};
void launch_xfwd8(const X8Job& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                  cudaStream_t s);
void launch_ycol(const YJob& job, const GridDims& g, const LineTables& ty, const DevStatus* st,
                 cudaStream_t s);

// species2d%cbq between the two x passes: y forward (times scale), the
// smoothing of every mode, y inverse, in one pass over the columns
void launch_ysmooth(const YJob& job, const GridDims& g, const KCoef& K, const LineTables& ty,
                    const DevStatus* st, cudaStream_t s);

}  // namespace qp
