// qp_misc.cuh -- launch interface of the solve, algebra, guard and glue kernels.
#pragma once

#include "qp_common.cuh"
#include "qp_solve.cuh"

namespace qp {

struct KPtrs {
  float* p[8];
};
struct Planes3 {
  float* p[3];
};

// Element-wise operations on planes, several planes per launch (grid row i =
// plane i).  Every plane starts on a 16-byte boundary and holds a multiple of
// four floats (field pitches and particle capacities are such); the planes of
// one job must not depend on one another (lin_conflict).
//   FILL d = v   SCALE d = a v   ADD d = a + b   SUB d = a - b   COPY d = a
//   ADD3 d = c + (a + b)         ADDSC d = a + b, then s = a v (s may be a)
enum { LIN_FILL = 0, LIN_SCALE, LIN_ADD, LIN_SUB, LIN_COPY, LIN_ADD3, LIN_ADDSC };
constexpr int LIN_MAX = 24;
struct LinPlane {
  float* d;
  const float* a;
  const float* b;
  const float* c;
  float* s;
  long long n;
  float v;
  int op;
};
struct LinJob {
  LinPlane p[LIN_MAX];
  int count;
};
// whether plane `q` reads or writes what a plane of the job writes, or writes
// what one of them reads: then it has to wait for them
bool lin_conflict(const LinJob& job, const LinPlane& q);
void launch_lin_job(const LinJob& job, const DevStatus* st, cudaStream_t s);

// A list of element-wise operations in the caller's order, launched in as few
// jobs as their dependences allow.  flush() returns the launches made so far.
class LinList {
 public:
  LinList(const DevStatus* st, cudaStream_t s) : st_(st), s_(s) {}
  void add(const LinPlane& q) {
    if (job_.count == LIN_MAX || lin_conflict(job_, q)) flush();
    job_.p[job_.count++] = q;
  }
  void add(int op, long long n, float* d, const float* a = nullptr, const float* b = nullptr,
           float v = 0.f) {
    add(LinPlane{d, a, b, nullptr, nullptr, n, v, op});
  }
  int flush() {
    if (job_.count) {
      launch_lin_job(job_, st_, s_);
      ++launches_;
    }
    job_.count = 0;
    return launches_;
  }

 private:
  LinJob job_{};
  int launches_ = 0;
  const DevStatus* st_;
  cudaStream_t s_;
};

void launch_lin(long long n, float* d, const float* a, const float* b, float v, int op,
                const DevStatus* st, cudaStream_t s);

// d = src[n-1] + (... + (src[0] + 0)), or on top of d when `onto` is set
constexpr int SUM_MAX = 16;
struct SumJob {
  const float* src[SUM_MAX];
  int count, onto;
};
void launch_sum(const SumJob& job, long long n, float* d, const DevStatus* st, cudaStream_t s);
// of `count` (1..3) planes in one launch
void launch_guard_copy(float* const* p, int count, const GridDims& g, const DevStatus* st,
                       cudaStream_t s);
void launch_guard_add(float* const* p, int count, const GridDims& g, const DevStatus* st,
                      cudaStream_t s);
// Between device planes and the caller's interleaved arrays: element
// c + dim (a + n0 b) of the host array is scale * src[c][b pitch + a stride]
// for b < n1 (and a < count[b] when count is given), 0 otherwise.
struct PackJob {
  float* plane[8];
  int dim;              // host extents: components,
  long long n0, n1;     //   fast index, slow index
  long long valid1;     // slow indices that have data
  int stride;           // floats between consecutive fast indices of a plane
  long long pitch;      // floats between consecutive slow indices of a plane
  const int* count;
  float scale;
};
// Where element i of the host array lies: component *c and the float of its
// plane; false for an element without data.
__host__ __device__ inline bool pack_at(const PackJob& j, long long i, int* c, long long* at) {
  const long long row = j.dim * j.n0, b = i / row, r = i - b * row, a = r / j.dim;
  *c = (int)(r - a * j.dim);
  *at = b * j.pitch + a * j.stride;
#ifdef __CUDA_ARCH__
  if (j.count && a >= j.count[b]) return false;
#endif
  return b < j.valid1;
}
// elements [i0, i0 + n) of the host array; `out` and `in` are pinned host (or
// device) memory and start at element i0.  No status check: a caller may look at
// the fields after an error.
void launch_pack(const PackJob& job, long long i0, long long n, float* out, cudaStream_t s);
// the reverse, data within valid1 and count only
void launch_unpack(const PackJob& job, long long i0, long long n, const float* in,
                   cudaStream_t s);
void launch_cursor(DevStatus* st, int v, cudaStream_t s);
}  // namespace qp
