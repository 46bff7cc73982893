// Device-side types and launchers shared by the engines.
#pragma once

#include <cuda_runtime.h>

#include "ctr_internal.h"

namespace ctr {

// One block GEMM task of the FP64 engine: C = sum_q w_q op(A_q) op(B_q).
struct ZTask {
  const double2* A[4];
  const double2* B[4];
  double2* C;
  float wre[4], wim[4];
  int nterm;
  int flags;  // bit q: conj-transpose A_q; bit 4+q: conj-transpose B_q
};

// One Hadamard trace: *out = coef * sum X (.) conj(Y)   (mode 0)
//                      *out = coef * Tr[X Y]            (mode 1)
// and, if absout is set, *absout = |coef| * sum |X_ij|_1 |Y_ij|_1 (mode 0) or
// |coef| * sum |X_ij|_1 |Y_ji|_1 (mode 1), |z|_1 = |Re z| + |Im z| (within a factor
// 2 of the product of moduli): the scale of the trace's rounding errors.
struct TraceTask {
  const double2* X;
  const double2* Y;
  double2* out;
  double* absout;
  float coef[2];
  int mode;  // bit 0: Y transposed (no conjugate); bit 1: the trace without its coefficient
  int pad;
};

__host__ __device__ inline double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// c += a b as four FMAs into the accumulator (the FP64 pipe is the bound of
// every caller)
__device__ inline void cmac(double2& c, double2 a, double2 b) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
}

// Sum over a 256-thread block with a fixed reduction tree (deterministic).
__device__ inline double block_sum_256(double v) {
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; w++) r += red[w];
  return r;  // valid in thread 0
}

// |c| of a row's coefficient; exact where it is real or imaginary, as the tables' are.
__device__ __forceinline__ double coef_abs(float re, float im) {
  if (im == 0.f) return fabs((double)re);
  if (re == 0.f) return fabs((double)im);
  return sqrt((double)re * re + (double)im * im);
}

// Block sums of two FP64 values: lanes 0-15 of each warp carry the first, 16-31
// the second (5 adds a warp instead of 10: each holds the FP64 pipe for 16
// clocks), then the warps' sums in order.  Thread k < 2 returns value k.
template <int TPB>
__device__ __forceinline__ double block_sum2(double x, double y) {
  __shared__ double red[TPB / 32][2];
  const int lane = threadIdx.x & 31;
  double s = ((lane & 16) ? y : x) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? x : y, 16);
  for (int o = 8; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((lane & 15) == 0) red[threadIdx.x >> 5][lane >> 4] = s;
  __syncthreads();
  double v = 0.0;
  if (threadIdx.x < 2) {
    v = red[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < TPB / 32; w++) v += red[w][threadIdx.x];
  }
  return v;
}

// h_tasks: the same tasks on the host (optional); it lets the launcher check
// that the weights allow the DMMA form.
int launch_zgemm_f64(const ZTask* d_tasks, int ntask, int N, cudaStream_t s, const ZTask* h_tasks = nullptr);
int launch_trace_f64(const TraceTask* d_tasks, int ntask, int N, cudaStream_t s);
// The launch alone, not counted or timed.
int launch_trace_f64_untimed(const TraceTask* d_tasks, int ntask, int N, cudaStream_t s);
// out[i * per + k] = (sum (|Re x| + |Im x|)^2)^(1/2) over the k-th of `per` consecutive blocks at base[i].
int launch_block_norms(const double2* const* d_base, int nbase, int per, int N, double* out, cudaStream_t s);
// loop[t] = sum_s Tr[tau(t,t)_ss Phi(t)] for diag [Nt][4][4][N][N], mom [Nt][N][N].
int launch_loop_unity(const double2* diag, const double2* mom, int N, int Nt, double2* loop, cudaStream_t s);
int launch_rowsum_coef(const double2* tr, int ntr, const int* off, const int* idx, const int* tix, const float* coef,
                       int nout, int npair, double2* out, cudaStream_t s);
int launch_source_average(int Nt, int ncorr, const double2* corr, double scale, double2* avg, cudaStream_t s);
// The same with per-entry refinement flags: entry p * nout + o of trace values and error
// scales tr, trabs [npair][ntr] is listed in list (+ pair_base * nout) and counted where
// eps_over_tol times its scale sum |coef| trabs exceeds its magnitude.
int launch_rowsum_coef_refine(const double2* tr, const double* trabs, int ntr, const int* off, const int* idx,
                              const int* tix, const float* coef, int nout, int npair, double2* out,
                              double eps_over_tol, int* count, int* list, int pair_base, cudaStream_t s);
// Scatter: out[where[i]] = vals[i].
int launch_scatter(const int* where, const double2* vals, int n, double2* out, cudaStream_t s);

}  // namespace ctr
