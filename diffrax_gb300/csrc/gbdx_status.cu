// gbdx_status.cu -- the outcome of a solve for the host in one launch: whether
// SaveAt's times were valid (diffrax/_integrate.py:1222-1235) and which trajectories
// failed (is_okay, diffrax/_solution.py:52-54).
//
// Bound: launch latency; the reads (4 bytes a trajectory, its interval when times
// are to be checked) are small beside a solve's.
#include "gbdx_launch.h"

namespace gbdx {
int set_last_error(int code, const char *msg);

namespace {

struct StatusScratch {  // all zero between calls
  unsigned long long first;  // ~(index << 8 | code) of the first failure, kept as a maximum
  unsigned int failed, outside, unsorted, ticket;
};

__global__ void __launch_bounds__(256) status_kernel(const int32_t *result, int64_t batch,
                                                     const double *t0, const double *t1,
                                                     int64_t time_stride, const double *ts,
                                                     int n_ts, StatusScratch *S, int32_t *out) {
  __shared__ double lo[256], hi[256];
  const int t = threadIdx.x;
  int falls = 0, rises = 0;
  double a = INFINITY, b = -INFINITY;
  for (int k = t; k < n_ts; k += 256) {
    const double x = ts[k];
    a = fmin(a, x);
    b = fmax(b, x);
    if (k > 0) {
      falls |= x < ts[k - 1];
      rises |= x > ts[k - 1];
    }
  }
  lo[t] = a;
  hi[t] = b;
  falls = __syncthreads_or(falls);
  rises = __syncthreads_or(rises);
  for (int n = 128; n; n /= 2) {
    if (t < n) {
      lo[t] = fmin(lo[t], lo[t + n]);
      hi[t] = fmax(hi[t], hi[t + n]);
    }
    __syncthreads();
  }
  const double tmin = lo[0], tmax = hi[0];
  unsigned int failed = 0;
  int outside = 0, unsorted = 0;
  unsigned long long first = 0;
  auto times = [&](double x, double y) {
    const bool up = x < y;  // else time runs backwards
    unsorted |= n_ts > 1 && (up ? falls : rises);
    outside |= up ? tmax > y || tmin < x : tmin < y || tmax > x;
  };
  if (n_ts > 0 && time_stride == 0 && blockIdx.x == 0 && t == 0) times(t0[0], t1[0]);
  for (int64_t i = int64_t(blockIdx.x) * 256 + t; i < batch; i += int64_t(gridDim.x) * 256) {
    if (n_ts > 0 && time_stride) times(t0[i * time_stride], t1[i * time_stride]);
    const int r = result ? result[i] : 0;
    if (r != GBDX_SUCCESSFUL && r != GBDX_EVENT_OCCURRED) {
      failed++;
      const unsigned long long key = ~((unsigned long long)i << 8 | (unsigned)(r & 255));
      first = first > key ? first : key;
    }
  }
  if (failed) {
    atomicAdd(&S->failed, failed);
    atomicMax(&S->first, first);
  }
  if (outside) S->outside = 1;
  if (unsorted) S->unsorted = 1;
  __threadfence();
  __syncthreads();
  if (t == 0 && atomicAdd(&S->ticket, 1u) == gridDim.x - 1) {
    __threadfence();
    volatile StatusScratch *V = S;
    out[0] = V->unsorted;
    out[1] = V->outside;
    out[2] = (int32_t)V->failed;
    out[3] = V->failed ? int32_t(~V->first & 255ull) : 0;
    V->first = 0;
    V->failed = V->outside = V->unsorted = V->ticket = 0;
  }
}

}  // namespace
}  // namespace gbdx

extern "C" int gbdx_solve_status(const int32_t *result, int64_t batch, const double *t0,
                                 const double *t1, int64_t time_stride, const double *ts,
                                 int32_t n_ts, void *scratch, int32_t *status, void *stream) {
  if (batch < 0 || n_ts < 0 || !scratch || !status || (n_ts > 0 && (!ts || !t0 || !t1)))
    return gbdx::set_last_error(GBDX_ERR_INVALID, "gbdx_solve_status: invalid argument");
  const int64_t want = (batch + 1023) / 1024;
  const int grid = int(want < 1 ? 1 : want > 64 ? 64 : want);
  gbdx::status_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      result, batch, t0, t1, time_stride, ts, n_ts, static_cast<gbdx::StatusScratch *>(scratch),
      status);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return gbdx::set_last_error(GBDX_ERR_CUDA, cudaGetErrorString(e));
  return GBDX_OK;
}
