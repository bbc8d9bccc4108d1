// qp_fft.cu -- 2D real sine/cosine transforms of field planes (x pass with an
// on-chip transpose, y pass on contiguous columns) and their twiddle tables.
//
// fftrk of a field (field2d_class.f03:157-191) = x pass over rows y = 0..ny
// writing the transposed [kx][y] array, then y pass over columns kx = 0..nx;
// the two passes together carry the reference's normalisation 0.25/(nx*ny).
// fftkr (field2d_class.f03:193-227) = the unnormalised y pass, then the x pass
// reading [kx][y] and writing rows, then the guard copy row ny = row 0
// (ufield2d copyguard, ufield2d_lib.f03:37-42) done by the CTA owning row 0.
#include <algorithm>
#include <cmath>
#include <vector>

#include "qp_fft.cuh"
#include "qp_line.cuh"

namespace qp {

int line_tables_build(LineTablesHost* t, int logn) {
  const int n = 1 << logn, h = n >> 1;
  std::vector<float> sn(n + 1), cs(n + 1);
  std::vector<float2> tw(h), uw(h + 1);
  const double pi = 3.14159265358979323846;
  for (int j = 0; j <= n; ++j) {
    sn[j] = (float)std::sin(pi * j / n);
    cs[j] = (float)std::cos(pi * j / n);
  }
  for (int m = 0; m < h; ++m)
    tw[m] = make_float2((float)std::cos(-2.0 * pi * m / h), (float)std::sin(-2.0 * pi * m / h));
  for (int k = 0; k <= h; ++k)
    uw[k] = make_float2((float)std::cos(-2.0 * pi * k / n), (float)std::sin(-2.0 * pi * k / n));
  // the per-lane rearrangement for the register transform (n >= 64)
  const int P = n >= 64 ? n / 64 : 0;
  std::vector<float> lt(lt_floats(P), 0.f);
  if (P > 0) {
    auto f2 = [&](int off, int i, float2 v) {
      lt[off + 2 * i] = v.x;
      lt[off + 2 * i + 1] = v.y;
    };
    auto brev5 = [](int v) {
      int r = 0;
      for (int b = 0; b < 5; ++b)
        if (v >> b & 1) r |= 1 << (4 - b);
      return r;
    };
    for (int a = 0; a < P; ++a)
      for (int l = 0; l < 32; ++l) {
        const int m = l + 32 * a, j0 = 2 * m, j1 = 2 * m + 1;
        // twice the sines and half the twiddles after the first DFT: the factor
        // 0.5 of the pre-twiddle costs nothing there (powers of two are exact)
        f2(lt_sn(P), 32 * a + l,
           make_float2(2.f * sn[std::min(j0, n - j0)], 2.f * sn[std::min(j1, n - j1)]));
        f2(lt_cs(P), 32 * a + l, make_float2(cs[j0], cs[j1]));
      }
    for (int k2 = 0; k2 < P; ++k2)
      for (int l = 0; l < 32; ++l) {
        const float2 t4 = tw[l * k2];
        f2(lt_tw4(P), 32 * k2 + l, make_float2(0.5f * t4.x, 0.5f * t4.y));
        f2(lt_uw(P), 32 * k2 + l, uw[k2 + P * (line_xs(P) ? l : brev5(l))]);
      }
    for (int si = 0; si < 4; ++si) {
      const int st = 16 >> si;
      for (int l = 0; l < 32; ++l)
        f2(lt_tw5(P), 32 * si + l,
           (l & st) ? tw[(l & (st - 1)) * (16 / st) * P] : make_float2(1.f, 0.f));
    }
    for (int k = 0; k < 16; ++k) f2(lt_tw3(P), k, tw[k * P]);
    // exp(-2 pi i q c / 32) = tw[q c P] for the exchange form's 8 x 4 split
    for (int q = 0; q < 4; ++q)
      for (int c = 0; c < 8; ++c) f2(lt_w32(P), 8 * q + c, tw[q * c * P]);
  }
  size_t bytes = sizeof(float) * 2 * (n + 1) + sizeof(float2) * (2 * h + 1) + 64 +
                 sizeof(float) * lt.size() + 16;
  char* d = nullptr;
  if (cudaMalloc(&d, bytes) != cudaSuccess) return -2;
  float* dsn = reinterpret_cast<float*>(d);
  float* dcs = dsn + (n + 1);
  size_t off = (sizeof(float) * 2 * (n + 1) + 15) & ~size_t(15);
  float2* dtw = reinterpret_cast<float2*>(d + off);
  float2* duw = dtw + h;
  cudaMemcpy(dsn, sn.data(), sizeof(float) * (n + 1), cudaMemcpyHostToDevice);
  cudaMemcpy(dcs, cs.data(), sizeof(float) * (n + 1), cudaMemcpyHostToDevice);
  cudaMemcpy(dtw, tw.data(), sizeof(float2) * h, cudaMemcpyHostToDevice);
  if (cudaMemcpy(duw, uw.data(), sizeof(float2) * (h + 1), cudaMemcpyHostToDevice) != cudaSuccess)
    return -2;
  float* dlt = nullptr;
  if (P > 0) {
    const size_t lo = ((size_t)(reinterpret_cast<char*>(duw + h + 1) - d) + 15) & ~size_t(15);
    dlt = reinterpret_cast<float*>(d + lo);
    if (cudaMemcpy(dlt, lt.data(), sizeof(float) * lt.size(), cudaMemcpyHostToDevice) !=
        cudaSuccess)
      return -2;
  }
  t->t.lane = dlt;
  t->t.lane_floats = (int)lt.size();
  t->base = d;
  t->t.sn = dsn;
  t->t.cs = dcs;
  t->t.tw = dtw;
  t->t.uw = duw;
  t->logn = logn;
  return 0;
}

void line_tables_free(LineTablesHost* t) {
  if (t->base) cudaFree(t->base);
  t->base = nullptr;
}

// ------------------------------------------------------------------ x pass
// The slice cursor must name one of the planes of the 3D array a component
// reads or writes; otherwise the launch raises an error and does nothing.
__device__ __forceinline__ bool cursor_ok(const XComp& c, const DevStatus* st) {
  const int cur = st->cursor + c.cursor_next;
  if (cur >= 0 && cur < c.cursor_planes) return true;
  if (threadIdx.x == 0) atomicCAS(const_cast<int*>(&st->error), 0, -7);
  return false;
}

// Shared memory of the line kernels: 8 lines of pitch n + 4 floats (16-byte
// aligned rows; the transposed accesses below hit 32 distinct banks), plus 8
// scratch lines for lines shorter than 64 points.
static __host__ __device__ int line_pitch(int n) { return n + 4; }
static __host__ __device__ int line_count(int logn) { return logn < 6 ? 16 : 8; }

// Forward x pass: for every component c and row y, the line
//   x[j] = scale_c * (src_c[y][j] + src2_c[y][j]),  j = 0..nx
// is transformed with parity_c and stored transposed into dst_c[kx][y].
// The 8 rows y0 .. y0 + 7 of component c (the CTA's 8 warps).
template <int P>
__device__ __forceinline__ void xfwd_rows(const XComp& c, int y0, const GridDims& g,
                                          const LineTables& tx, float* smem, float* T,
                                          const DevStatus* st) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = g.nx, pitch = line_pitch(n);
  float* L = smem + warp * pitch;
  float* S = smem + (8 + warp) * pitch;
  const int y = y0 + warp;
  const long long cur =
      c.cursor_stride ? (long long)(st->cursor + c.cursor_next) * c.cursor_stride : 0;
  if (P > 0) __syncthreads();
  if (y <= g.ny) {
    const float* s1 = c.src + cur + (long long)y * g.rp;
    const float* s2 = c.src2 ? c.src2 + (long long)y * g.rp : nullptr;
    line_transform<P>(s1, s2, c.scale, L, S, g.indx, c.parity, tx, T, lane);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < (n + 1) * 8; idx += 256) {
    const int r = idx & 7, kx = idx >> 3;
    const int yy = y0 + r;
    if (yy <= g.ny) c.dst[(long long)kx * g.kp + yy] = smem[r * pitch + kx];
  }
}

template <int P>
__global__ void __launch_bounds__(256) k_xfwd(XJob job, GridDims g, LineTables tx,
                                              const DevStatus* st) {
  extern __shared__ __align__(16) float smem[];
  float* T = smem + line_count(g.indx) * line_pitch(g.nx);
  if (P > 0) stage_lane_table(T, tx);  // constant tables: staged before the wait
  grid_dep_sync();
  if (st && st->error) return;
  const XComp c = job.c[blockIdx.y];
  if (c.cursor_stride && !cursor_ok(c, st)) return;
  xfwd_rows<P>(c, blockIdx.x * 8, g, tx, smem, T, st);
}

// Inverse x pass: rows y of the [kx][y] array are gathered, transformed with
// parity_c, scaled and written as real-space rows; row 0 is also written to the
// guard row ny (copyguard), and the line computed for row ny is discarded.
// The 8 rows y0 .. y0 + 7 of component c (the CTA's 8 warps).
template <int P>
__device__ __forceinline__ void xinv_rows(const XComp& c, int y0, const GridDims& g,
                                          const LineTables& tx, float* smem, float* T,
                                          const DevStatus* st) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = g.nx, pitch = line_pitch(n);
  // the 8 rows' [kx][y] entries, 32 bytes per kx: batches of 8 loads per
  // thread are all issued before their shared-memory stores, so a thread waits
  // for L2 twice per 16 loads instead of once per load
  const int total = (n + 1) * 8;
  for (int b0 = threadIdx.x; b0 < total; b0 += 8 * 256) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = b0 + u * 256;
      const int yy = y0 + (idx & 7);
      v[u] = (idx < total && yy <= g.ny) ? c.src[(long long)(idx >> 3) * g.kp + yy] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = b0 + u * 256;
      if (idx < total) smem[(idx & 7) * pitch + (idx >> 3)] = v[u];
    }
  }
  __syncthreads();
  float* L = smem + warp * pitch;
  float* S = smem + (8 + warp) * pitch;
  const int y = y0 + warp;
  if (y < g.ny) {
    line_transform<P>(L, nullptr, 1.f, L, S, g.indx, c.parity, tx, T, lane);
    long long cur = 0;
    if (c.cursor_stride) cur = (long long)(st->cursor + c.cursor_next) * c.cursor_stride;
    float* d = c.dst + cur + (long long)y * g.rp;
    line_store(d, L, n, c.scale, lane);
    if (y == 0) {
      float* dg = c.dst + cur + (long long)g.ny * g.rp;
      line_store(dg, L, n, c.scale, lane);
      if (lane == 0) dg[n + 1] = d[n + 1];
    }
  }
}

template <int P>
__global__ void __launch_bounds__(256) k_xinv(XJob job, GridDims g, LineTables tx,
                                              const DevStatus* st) {
  extern __shared__ __align__(16) float smem[];
  const int pitch = line_pitch(g.nx);
  float* T = smem + line_count(g.indx) * pitch;
  // constant tables, staged before the wait; the barrier after the gather covers them
  if (P > 0) stage_lane_table(T, tx);
  grid_dep_sync();
  if (st && st->error) return;
  const XComp c = job.c[blockIdx.y];
  if (c.cursor_stride && !cursor_ok(c, st)) return;
  const int y0 = blockIdx.x * 8;
  xinv_rows<P>(c, y0, g, tx, smem, T, st);
}

// Inverse x pass of node-major fields.  A CTA takes two rows of one group of
// four components, its warps one line each: a (kx, y) pair of rows is one
// 32-byte sector of the [kx][y][4] array, read as two float4, and a node of the
// result is one float4 of the [y][x][4] array -- 5 loads and 5 stores of 16
// bytes per thread at 512 points, where the planar form makes 17 of 4 bytes
// each.  The remaining CTAs transform planar components, 8 rows each.
// Bound by latency and the transforms' shared-memory and shuffle traffic: 14.2
// -> 14.0 us at 512 x 512 (five components).
template <int P>
__global__ void __launch_bounds__(256) k_xinv4(const __grid_constant__ X4Job job, GridDims g,
                                               LineTables tx, const DevStatus* st) {
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = g.nx, pitch = line_pitch(n);
  float* T = smem + line_count(g.indx) * pitch;
  if (P > 0) stage_lane_table(T, tx);  // constant tables: staged before the wait
  grid_dep_wait();
  if (!job.hold) grid_dep_launch();
  if (st && st->error) return;
  if (pass_skipped(st, job.pass)) return;
  float* L = smem + warp * pitch;
  float* S = smem + (8 + warp) * pitch;
  const int pairs = g.ny >> 1;
  if ((int)blockIdx.x < job.ngroup * pairs) {
    const int gi = (int)blockIdx.x >= pairs ? 1 : 0;
    const int y0 = 2 * ((int)blockIdx.x - gi * pairs);
    const float4* src = job.src[gi] + y0;
    // node (kx, row r) -> lines 4 r .. 4 r + 3; every load before the stores (5 a
    // thread are the 1026 of a 512-point line; longer lines take rounds of 4)
    constexpr int U = P == 8 ? 5 : 4;
    const int total = 2 * (n + 1);
    for (int b0 = threadIdx.x; b0 < total; b0 += U * 256) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b0 + u * 256;
        if (i < total) v[u] = src[(long long)(i >> 1) * g.kp + (i & 1)];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b0 + u * 256;
        if (i < total) {
          float* d = smem + 4 * (i & 1) * pitch + (i >> 1);
          d[0] = v[u].x;
          d[pitch] = v[u].y;
          d[2 * pitch] = v[u].z;
          d[3 * pitch] = v[u].w;
        }
      }
    }
    __syncthreads();
    line_transform<P>(L, nullptr, 1.f, L, S, g.indx, job.par[gi][warp & 3], tx, T, lane);
    __syncthreads();
    for (int r = 0; r < 2; ++r) {
      float4* d = job.dst[gi] + (long long)(y0 + r) * g.rp;
      const float* l = smem + 4 * r * pitch;
      for (int i = threadIdx.x; i <= n; i += 256) {
        const float4 v = node4(l, pitch, i);
        d[i] = v;
        if (y0 + r == 0) job.dst[gi][(long long)g.ny * g.rp + i] = v;  // copyguard
      }
    }
  } else {
    const int b = (int)blockIdx.x - job.ngroup * pairs, per = g.ny >> 3;
    const XComp c = job.x.c[b / per];
    if (c.cursor_stride && !cursor_ok(c, st)) return;
    xinv_rows<P>(c, 8 * (b % per), g, tx, smem, T, st);
  }
  // the zero planes, a share per CTA (planes are multiples of 16 bytes)
  const long long n4 = g.rplane >> 2, share = (n4 + gridDim.x - 1) / gridDim.x;
  const long long lo = share * blockIdx.x, hi = min(n4, lo + share);
  for (int z = 0; z < job.nzero; ++z)
    for (long long i = lo + threadIdx.x; i < hi; i += 256)
      reinterpret_cast<float4*>(job.zero[z])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Forward x pass of node-major densities.  A CTA takes one row, its 8 warps
// the 8 components: the row is one run of 16-byte loads, which the warps
// spread over 8 shared lines (lane pairs take a node: component 4 h + k of
// node i goes to bank 16 h + 4 k + i, so no two lanes of a store collide), and
// a node of the transposed result is one full 32-byte sector -- 5 loads and 5
// stores of 16 bytes per thread at 512 points, where the planar form loads 8
// bytes and stores 4 at a time.  Planar components follow, 8 rows per CTA.
// Bound by the transforms' shared-memory and shuffle traffic: 14.7 us at 512 x
// 512 (9.4 MB in and out); the planar form took 13.3, the staging through
// shared memory being the price of the densities' vector reductions (amjdp
// 2.3 us less per pass).
// Registers per thread (resident CTAs) by line length: a cap pays where it
// makes room for one CTA more, 64 at 512 points (4 CTAs: 14.2 us, uncapped
// 14.4) and 80 at 1024 points (3 CTAs: 34.6 us with 36 bytes spilled, uncapped
// 35.6).  48 at 512 points (5 CTAs) would suit 64 concurrent instances (7.07 ->
// 7.15e9 particle-slices/s) but not one (4.48 -> 4.33e9).  Shorter lines take
// what they need (0): a cap makes the compiler spend registers up to it.  2048
// points leave one CTA per SM with any cap that does not spill heavily.
template <int P>
__global__ void __launch_bounds__(256, P == 8 ? 4 : P == 16 ? 3 : 0)
    k_xfwd8(const __grid_constant__ X8Job job, GridDims g, LineTables tx, const DevStatus* st) {
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = g.nx, pitch = line_pitch(n);
  float* T = smem + line_count(g.indx) * pitch;
  if (P > 0) stage_lane_table(T, tx);  // constant tables: staged before the wait
  grid_dep_sync();
  if (st && st->error) return;
  if (pass_skipped(st, job.pass)) return;
  if ((int)blockIdx.x >= g.ny) {
    const int b = (int)blockIdx.x - g.ny, per = (g.ny + 8) >> 3;
    const XComp c = job.x.c[b / per];
    if (c.cursor_stride && !cursor_ok(c, st)) return;
    xfwd_rows<P>(c, 8 * (b % per), g, tx, smem, T, st);
    return;
  }
  const int y = blockIdx.x;
  stage_lines8<P>(job.src + 2LL * y * g.rp, n, pitch, smem, 256);
  __syncthreads();
  float* L = smem + warp * pitch;
  float* S = smem + (8 + warp) * pitch;
  line_transform<P>(L, nullptr, 1.f, L, S, g.indx, job.par[warp], tx, T, lane);
  __syncthreads();
  float4* d = job.dst + 2LL * y;
  for (int i = threadIdx.x; i < 2 * (n + 1); i += 256)
    d[2LL * (i >> 1) * g.kp + (i & 1)] = node4(smem + 4 * (i & 1) * pitch, pitch, i >> 1);
}

// ------------------------------------------------------------------ y pass
// In-place y transform of the columns kx of component blockIdx.y, times
// scale_c; with SMOOTH the smoothing operator is applied to the transformed
// column and the column is transformed back (sine lines: parity_c of the
// inverse is that of the forward transform).  One warp per column and
// component: a launch is one latency chain (load, transform, store), so the
// components of a vector run side by side instead of one after another.
// 1024-point lines: registers capped at 80 (3 CTAs per SM); left alone the
// compiler takes 64, and a transform pair of one component at 1024 x 1024 takes
// 40.4 us instead of 24.9 (three components 62.9, 52.2).  Plain transforms of up
// to 256 points do not let the next grid in early: with several components they
// are more CTAs than SMs, and the x pass that follows has the long chains (1024
// x 64, two components: 24.9 -> 19.3 us a pair).  Longer ones gain from it (512 x
// 512, three components: 22.5 us against 23.5), and so does the smoothing of a
// step of two species (3.34 ms against 3.41 for 32 slices at 256 x 256).
template <int P, bool SMOOTH>
__global__ void __launch_bounds__(256, P == 16 ? 3 : 0) k_ycol(const __grid_constant__ YJob job, GridDims g,
                                              KCoef K, LineTables ty, const DevStatus* st) {
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = g.ny, pitch = line_pitch(n);
  float* L = smem + warp * pitch;
  float* S = smem + (8 + warp) * pitch;
  float* T = smem + line_count(g.indy) * pitch;
  if (P > 0) stage_lane_table(T, ty);  // constant tables: staged before the wait
  grid_dep_wait();
  if (SMOOTH || P == 0 || P >= 8) grid_dep_launch();
  if (st && st->error) return;
  if (P > 0) __syncthreads();
  const int kx = blockIdx.x * 8 + warp;
  if (kx > g.nx) return;
  const YComp c = job.c[blockIdx.y];
  float* col = c.plane + (long long)kx * g.kp;
  line_transform<P>(col, nullptr, 1.f, L, S, g.indy, c.parity, ty, T, lane);
  float scale = c.scale;
  if (SMOOTH) {
    for (int ky = lane; ky <= n; ky += 32) L[ky] = k_smooth(K, kx, ky, QM(L[ky], scale));
    __syncwarp();
    line_transform<P>(L, nullptr, 1.f, L, S, g.indy, c.parity, ty, T, lane);
    scale = 1.f;
  }
  line_store(col, L, n, scale, lane);
}

size_t xpass_smem(const GridDims& g) {
  return sizeof(float) * ((size_t)line_count(g.indx) * line_pitch(g.nx) + lt_floats(line_p(g.indx)));
}
size_t ypass_smem(const GridDims& g) {
  return sizeof(float) * ((size_t)line_count(g.indy) * line_pitch(g.ny) + lt_floats(line_p(g.indy)));
}

template <int P>
static int set_smem_limits(int big) {
  if (cudaFuncSetAttribute(k_xfwd<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_xinv<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_xfwd8<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_xinv4<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_ycol<P, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_ycol<P, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big) !=
          cudaSuccess)
    return -2;
  return 0;
}

int fft_kernels_init() {
  const int big = (int)(sizeof(float) * (8 * line_pitch(1 << QP_MAX_IND) +
                                         lt_floats(line_p(QP_MAX_IND))));
  for (int logn = 4; logn <= QP_MAX_IND; ++logn) {
    int rc = 0;
    QP_LINE_SWITCH(logn, rc = set_smem_limits<P_>(big));
    if (rc) return rc;
  }
  return 0;
}

void launch_xfwd(const XJob& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                 cudaStream_t s) {
  dim3 grid((g.ny + 1 + 7) / 8, job.ncomp);
  QP_LINE_SWITCH(g.indx, (launch_pdl(k_xfwd<P_>, grid, 256, xpass_smem(g), s, job, g, tx, st)));
}

void launch_xinv(const XJob& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                 cudaStream_t s) {
  dim3 grid((g.ny + 1 + 7) / 8, job.ncomp);
  QP_LINE_SWITCH(g.indx, (launch_pdl(k_xinv<P_>, grid, 256, xpass_smem(g), s, job, g, tx, st)));
}

void launch_xfwd8(const X8Job& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                  cudaStream_t s) {
  const int grid = g.ny + job.x.ncomp * ((g.ny + 8) >> 3);
  QP_LINE_SWITCH(g.indx, (launch_pdl(k_xfwd8<P_>, grid, 256, xpass_smem(g), s, job, g, tx, st)));
}

void launch_xinv4(const X4Job& job, const GridDims& g, const LineTables& tx, const DevStatus* st,
                  cudaStream_t s) {
  const int grid = job.ngroup * (g.ny >> 1) + job.x.ncomp * (g.ny >> 3);
  QP_LINE_SWITCH(g.indx, (launch_pdl(k_xinv4<P_>, grid, 256, xpass_smem(g), s, job, g, tx, st)));
}

void launch_ycol(const YJob& job, const GridDims& g, const LineTables& ty, const DevStatus* st,
                 cudaStream_t s) {
  dim3 grid((g.nx + 1 + 7) / 8, job.ncomp);
  QP_LINE_SWITCH(g.indy, (launch_pdl(k_ycol<P_, false>, grid, 256, ypass_smem(g), s, job, g,
                                     KCoef{}, ty, st)));
}

void launch_ysmooth(const YJob& job, const GridDims& g, const KCoef& K, const LineTables& ty,
                    const DevStatus* st, cudaStream_t s) {
  dim3 grid((g.nx + 1 + 7) / 8, job.ncomp);
  QP_LINE_SWITCH(g.indy, (launch_pdl(k_ycol<P_, true>, grid, 256, ypass_smem(g), s, job, g, K, ty,
                                     st)));
}

}  // namespace qp
