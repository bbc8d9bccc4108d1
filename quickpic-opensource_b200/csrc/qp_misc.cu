// qp_misc.cu -- Fourier-space solve kernels, field algebra, guard operations
// and the small per-slice kernels of the fused 3D step.
#include "qp_misc.cuh"

#include <algorithm>

namespace qp {

namespace {

__device__ __forceinline__ bool kidx(const GridDims& g, int i, int* kx, int* ky) {
  const int n1 = g.ny + 1;
  if (i >= (g.nx + 1) * n1) return false;
  *kx = i / n1;
  *ky = i - *kx * n1;
  return true;
}

__global__ void k_kpoint(int op, GridDims g, KCoef K, KPtrs in, KPtrs out, float aa, float dex,
                         const DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  int kx, ky;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (!kidx(g, i, &kx, &ky)) return;
  const long long o = (long long)kx * g.kp + ky;
  switch (op) {
    case KOP_POT:
      out.p[0][o] = k_pot(K, kx, ky, in.p[0][o]);
      break;
    case KOP_SMOOTH:
      out.p[0][o] = k_smooth(K, kx, ky, in.p[0][o]);
      break;
    case KOP_ELF: {
      float fx, fy;
      k_elf(K, kx, ky, in.p[0][o], &fx, &fy);
      out.p[0][o] = fx;
      out.p[1][o] = fy;
      break;
    }
    case KOP_BF: {
      float bx, by, bz;
      k_bf(K, kx, ky, in.p[0][o], in.p[1][o], in.p[2][o], &bx, &by, &bz);
      out.p[0][o] = bx;
      out.p[1][o] = by;
      out.p[2][o] = bz;
      break;
    }
    case KOP_BFQP: {
      // in: cu(3), dcu(2) (in/out), amu(3); out: bxy(2) (in/out)
      float dcx = in.p[3][o], dcy = in.p[4][o];
      float bx = out.p[0][o], by = out.p[1][o];
      k_bfqp(K, kx, ky, aa, 1.f / dex, in.p[2][o], &dcx, &dcy, in.p[5][o], in.p[6][o],
             in.p[7][o], &bx, &by);
      in.p[3][o] = dcx;
      in.p[4][o] = dcy;
      out.p[0][o] = bx;
      out.p[1][o] = by;
      break;
    }
    case KOP_DIV:
      out.p[0][o] = k_div(K, kx, ky, in.p[0][o], in.p[1][o]);
      break;
    case KOP_GRAD: {
      float fx, fy;
      k_grad(K, kx, ky, in.p[0][o], &fx, &fy);
      out.p[0][o] = fx;
      out.p[1][o] = fy;
      break;
    }
    case KOP_VPOT: {
      float ax, ay, az;
      k_vpot(K, kx, ky, in.p[0][o], in.p[1][o], in.p[2][o], &ax, &ay, &az);
      out.p[0][o] = ax;
      out.p[1][o] = ay;
      out.p[2][o] = az;
      break;
    }
  }
}

__device__ __forceinline__ float lin1(int op, float a, float b, float c, float v) {
  switch (op) {
    case LIN_FILL: return v;
    case LIN_SCALE: return a * v;
    case LIN_SUB: return a - b;
    case LIN_COPY: return a;
    case LIN_ADD3: return c + (a + b);
    default: return a + b;  // LIN_ADD, LIN_ADDSC
  }
}

// One row of CTAs per plane, four nodes per thread and step.  Bound by launch
// latency: a plane is 0.02 - 4.2 MB and stays in L2, so a launch costs about
// 4 us in a stream whatever it moves.  What counts is the number of launches
// (the class interface's amjdp: 20 with one plane each, 3 with a job's).
__global__ void __launch_bounds__(256) k_lin(const __grid_constant__ LinJob job, const DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  const LinPlane& p = job.p[blockIdx.y];
  const int op = p.op;
  const float v = p.v;
  const bool ra = op != LIN_FILL, rb = op != LIN_FILL && op != LIN_SCALE && op != LIN_COPY;
  const bool rc = op == LIN_ADD3;
  const long long n4 = p.n >> 2;
  const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = i0; i < n4; i += step) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a = ra ? reinterpret_cast<const float4*>(p.a)[i] : z;
    const float4 b = rb ? reinterpret_cast<const float4*>(p.b)[i] : z;
    const float4 c = rc ? reinterpret_cast<const float4*>(p.c)[i] : z;
    reinterpret_cast<float4*>(p.d)[i] =
        make_float4(lin1(op, a.x, b.x, c.x, v), lin1(op, a.y, b.y, c.y, v),
                    lin1(op, a.z, b.z, c.z, v), lin1(op, a.w, b.w, c.w, v));
    if (op == LIN_ADDSC)
      reinterpret_cast<float4*>(p.s)[i] = make_float4(a.x * v, a.y * v, a.z * v, a.w * v);
  }
}

__global__ void __launch_bounds__(256) k_sum(const __grid_constant__ SumJob job, long long n,
                                             float* d, const DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  const long long n4 = n >> 2;
  const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = i0; i < n4; i += step) {
    float4 v = job.onto ? reinterpret_cast<const float4*>(d)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < job.count; ++k) {
      const float4 a = reinterpret_cast<const float4*>(job.src[k])[i];
      v = make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
    }
    reinterpret_cast<float4*>(d)[i] = v;
  }
}

// copyguard: row ny = row 0, every column (ufield2d_lib.f03:37-42)
__global__ void k_guard_copy(Planes3 pl, GridDims g, const DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  float* p = pl.p[blockIdx.y];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j <= g.nx + 1) p[(long long)g.ny * g.rp + j] = p[j];
}

// acopyguard: row 0 += row ny, row ny = 0 for columns 0..nx (ufield2d_lib.f03:90-97)
__global__ void k_guard_add(Planes3 pl, GridDims g, const DevStatus* st) {
  grid_dep_sync();
  if (st && st->error) return;
  float* p = pl.p[blockIdx.y];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j <= g.nx) {
    float* top = p + (long long)g.ny * g.rp + j;
    p[j] = p[j] + *top;
    *top = 0.f;
  }
}

// One host element per thread and step.  The host side is contiguous and, for
// the transfers of the C ABI, pinned host memory: the kernel itself moves the
// data over PCIe, in place of a copy of each plane and a strided loop on the
// host (2 ms per 512 x 512 vector; bound now by the host's page faults on the
// caller's fresh array, 1 us per 4 KB).
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackJob j, long long i0,
                                              long long n, float* out) {
  grid_dep_sync();
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    int c;
    long long at;
    out[k] = pack_at(j, i0 + k, &c, &at) ? j.plane[c][at] * j.scale : 0.f;
  }
}

__global__ void __launch_bounds__(256) k_unpack(const __grid_constant__ PackJob j, long long i0,
                                                long long n, const float* in) {
  grid_dep_sync();
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    int c;
    long long at;
    if (pack_at(j, i0 + k, &c, &at)) j.plane[c][at] = in[k];
  }
}

__global__ void k_cursor(DevStatus* st, int v) {
  grid_dep_sync();
  if (st->error) return;
  st->cursor = v;
}

}  // namespace

int launch_kpoint(int op, const GridDims& g, const KCoef& K, float* const* in, float* const* out,
                  float aa, float dex, const DevStatus* st, cudaStream_t s) {
  KPtrs a{}, b{};
  for (int i = 0; i < 8; ++i) {
    a.p[i] = in ? in[i] : nullptr;
    b.p[i] = out ? out[i] : nullptr;
  }
  const int n = (g.nx + 1) * (g.ny + 1);
  launch_pdl(k_kpoint, (n + 255) / 256, 256, 0, s, op, g, K, a, b, aa, dex, st);
  return 0;
}

bool lin_conflict(const LinJob& job, const LinPlane& q) {
  auto overlap = [](const float* x, long long nx, const float* y, long long ny) {
    return x && y && x < y + ny && y < x + nx;
  };
  for (int i = 0; i < job.count; ++i) {
    const LinPlane& p = job.p[i];
    for (const float* w : {(const float*)p.d, (const float*)p.s})
      for (const float* r : {(const float*)q.d, (const float*)q.s, q.a, q.b, q.c})
        if (overlap(w, p.n, r, q.n)) return true;
    for (const float* w : {(const float*)q.d, (const float*)q.s})
      for (const float* r : {p.a, p.b, p.c})
        if (overlap(w, q.n, r, p.n)) return true;
  }
  return false;
}

static int lin_blocks(long long n, int rows) {
  const long long want = ((n >> 2) + 255) / 256, most = std::max(1, 148 * 16 / rows);
  return (int)std::max(1LL, std::min(want, most));
}

void launch_lin_job(const LinJob& job, const DevStatus* st, cudaStream_t s) {
  long long n = 1;
  for (int i = 0; i < job.count; ++i) n = std::max(n, job.p[i].n);
  launch_pdl(k_lin, dim3(lin_blocks(n, job.count), job.count), 256, 0, s, job, st);
}

void launch_lin(long long n, float* d, const float* a, const float* b, float v, int op,
                const DevStatus* st, cudaStream_t s) {
  LinJob job{};
  job.p[0] = LinPlane{d, a, b, nullptr, nullptr, n, v, op};
  job.count = 1;
  launch_lin_job(job, st, s);
}

void launch_sum(const SumJob& job, long long n, float* d, const DevStatus* st, cudaStream_t s) {
  launch_pdl(k_sum, lin_blocks(n, 1), 256, 0, s, job, n, d, st);
}

static Planes3 planes3(float* const* p, int count) {
  Planes3 r{};
  for (int i = 0; i < count; ++i) r.p[i] = p[i];
  return r;
}

void launch_guard_copy(float* const* p, int count, const GridDims& g, const DevStatus* st,
                       cudaStream_t s) {
  launch_pdl(k_guard_copy, dim3((g.nx + 2 + 255) / 256, count), 256, 0, s, planes3(p, count), g,
             st);
}

void launch_guard_add(float* const* p, int count, const GridDims& g, const DevStatus* st,
                      cudaStream_t s) {
  launch_pdl(k_guard_add, dim3((g.nx + 1 + 255) / 256, count), 256, 0, s, planes3(p, count), g,
             st);
}

static int pack_blocks(long long n) {
  return (int)std::max(1LL, std::min((n + 255) / 256, 148LL * 8));
}

void launch_pack(const PackJob& job, long long i0, long long n, float* out, cudaStream_t s) {
  launch_pdl(k_pack, pack_blocks(n), 256, 0, s, job, i0, n, out);
}

void launch_unpack(const PackJob& job, long long i0, long long n, const float* in,
                   cudaStream_t s) {
  launch_pdl(k_unpack, pack_blocks(n), 256, 0, s, job, i0, n, in);
}

void launch_cursor(DevStatus* st, int v, cudaStream_t s) {
  launch_pdl(k_cursor, 1, 1, 0, s, st, v);
}

}  // namespace qp
