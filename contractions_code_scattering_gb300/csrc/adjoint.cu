// Distillation-profile adjoint: gradients of diagram traces with respect to a
// per-eigenvector profile f, where every elemental Phi(t, op) enters the
// contractions as diag(f) Phi diag(f).
//
// A chain is Tr[F_1 F_2 ... F_n] (2 <= n <= CTR_CHAIN_MAXF); each factor is a
// perambulator block tau(t1,t2)_{s1 s2} or a profiled elemental
// Phi'(t, op) = D Phi(t, op) D (D = diag f), either optionally
// conjugate-transposed.  For complex chain weights w_c the kernels compute
//   value_c = Tr[chain_c]   and   grad_k += Re sum_c w_c d value_c / d f_k.
//
// Reverse mode with recomputed prefix/suffix products.  With
// P_j = F_1 ... F_j and S_j = F_j ... F_n, the derivative of a trace at one
// occurrence of D is the diagonal of the cyclic product that starts right
// after it, d Tr[..D..]/d f_k = (rest)_kk, i.e. the transposed cyclic
// co-factor (F_{j+1}...F_n F_1...F_{j-1})^T of the adjoint of a product.  A
// profiled elemental F_j holds two D's, which gives
//   f_k d/df_k Tr = sum over elementals j of [diag(S_j P_{j-1}) + diag(S_{j+1} P_j)]_k
// with P_0 = S_{n+1} = identity.  Every diag(X Y) is an O(N^2) reduction
// (diag_reduce_kernel); the only GEMMs are the n-2 prefix and n-2 suffix
// products.  They are recomputed for every call (nothing from the forward
// pass is stored) and shared between chains by hash-consing: a prefix node is
// keyed by (parent, factor), a suffix node by (factor, child), so chains with
// a common head or tail (the spin rows of one diagram, the source times of
// one sink time) compute it once.  Nodes of equal depth form one batched GEMM
// launch.  The profile must have f_k != 0 (the diagonal identity above
// yields f_k d/df_k).
//
// The generic chains (ctr_chain_adjoint) run that way.  The diagrams' own gradients
// (rho: lib/calculate_rho_core.h; pi pi: lib/calculate_pipi_{square,
// doubleTriangle,doubleTriangleHor,starfish}_core.h) use their spin structure
// instead of one chain per spin row: a rho trace is Tr[A B] twice, cut at its
// two pairs of elementals, and the pi pi diagrams are traces of 4x4 spin-block
// matrices whose co-factors are a few four-term block products a pair (below).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "chains.h"

namespace ctr {

namespace {

// ------------------------------------------------------------------ kernels
// dst[m] = diag(f) src[m] diag(f), optionally for a strided subset.
__global__ void apply_profile_kernel(const double2* __restrict__ src, double2* __restrict__ dst,
                                     const double* __restrict__ f, int N, long long nmat) {
  const long long n = nmat * N * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int ij = (int)(e % ((long long)N * N));
    const double s = f[ij / N] * f[ij % N];
    const double2 v = src[e];
    dst[e] = make_double2(v.x * s, v.y * s);
  }
}

// One diagonal reduction d_k = sum_m op(X)[k][m] op(Y)[m][k]: buf[out * N + k] = Re(w d_k)
// where out >= 0 (w times *wp where wp is set), vals[vout] = sum_k d_k where vout >= 0.
struct DiagTask {
  const double2* x;
  const double2* y;
  const double2* wp;
  double wre, wim;
  int xdag, ydag;
  int out, vout;
};

__device__ __forceinline__ double2 diag_weight(const DiagTask& T) {
  const double2 w = make_double2(T.wre, T.wim);
  return T.wp ? cmul(w, *T.wp) : w;
}

// Nev <= 128.  The FP64 pipe is the bound (4 FMAs an element), so every lane of
// the working warps has an element: thread t takes k = t mod N and one of P
// (the largest divisor of DK with P N <= threads) shares of each chunk of DK m's,
// where 32-wide tiles padded N to a multiple of 32 (Nev = 100: 128).  X and Y go
// through shared memory in chunks of DK, read along their rows whatever the
// transposes.  Per task and SM at Nev = 100: see launch_diag.
constexpr int DIAG_TPB = 320, DK = 12;

__global__ void __launch_bounds__(DIAG_TPB) diag_small_kernel(const DiagTask* __restrict__ tasks, int N, int P,
                                                              double* __restrict__ buf, double2* __restrict__ vals) {
  extern __shared__ __align__(16) double2 dsm[];
  double2* xs = dsm;                 // [N][DK + 1]: op(X)[k][m0 + mm]
  double2* ys = xs + N * (DK + 1);   // [DK][N + 1]: op(Y)[m0 + mm][k]
  const DiagTask T = tasks[blockIdx.x];
  const int k = threadIdx.x % N, part = threadIdx.x / N, share = DK / P;
  const bool on = part < P;
  double2 acc = make_double2(0.0, 0.0);
  for (int m0 = 0; m0 < N; m0 += DK) {
    const int mn = min(DK, N - m0);
    for (int e = threadIdx.x; e < N * mn; e += DIAG_TPB) {
      {
        const int kk = T.xdag ? e % N : e / mn, mm = T.xdag ? e / N : e % mn;
        double2 v = T.xdag ? T.x[(size_t)(m0 + mm) * N + kk] : T.x[(size_t)kk * N + m0 + mm];
        if (T.xdag) v.y = -v.y;
        xs[kk * (DK + 1) + mm] = v;
      }
      {
        const int kk = T.ydag ? e / mn : e % N, mm = T.ydag ? e % mn : e / N;
        double2 v = T.ydag ? T.y[(size_t)kk * N + m0 + mm] : T.y[(size_t)(m0 + mm) * N + kk];
        if (T.ydag) v.y = -v.y;
        ys[mm * (N + 1) + kk] = v;
      }
    }
    __syncthreads();
    if (on) {
      const int hi = min(mn, (part + 1) * share);
      for (int mm = part * share; mm < hi; mm++) cmac(acc, xs[k * (DK + 1) + mm], ys[mm * (N + 1) + k]);
    }
    __syncthreads();
  }
  double2* part_sum = dsm;  // [P][N]
  if (on) part_sum[part * N + k] = acc;
  __syncthreads();
  double2 d = make_double2(0.0, 0.0);
  if (threadIdx.x < N) {
    d = part_sum[k];
    for (int q = 1; q < P; q++) {
      d.x += part_sum[q * N + k].x;
      d.y += part_sum[q * N + k].y;
    }
    if (T.out >= 0) {
      const double2 w = diag_weight(T);
      buf[(size_t)T.out * N + k] = w.x * d.x - w.y * d.y;
    }
  }
  if (T.vout >= 0) {
    const double v = block_sum2<DIAG_TPB>(d.x, d.y);
    if (threadIdx.x < 2) ((double*)(vals + T.vout))[threadIdx.x] = v;
  }
}

// Any Nev.  One CTA per task; 32x32 tiles of op(X) (rows k) and op(Y) (columns k)
// are staged through shared memory with coalesced reads whatever the transposes,
// so both operands are read once.
__global__ void __launch_bounds__(256) diag_reduce_kernel(const DiagTask* __restrict__ tasks, int N,
                                                          double* __restrict__ buf, double2* __restrict__ vals) {
  __shared__ double2 xs[32][33];
  __shared__ double2 ys[32][33];
  __shared__ double2 part[8][32];
  __shared__ double2 tot[32];
  const DiagTask T = tasks[blockIdx.x];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double2 vsum = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < N; k0 += 32) {
    double2 acc = make_double2(0.0, 0.0);  // thread (tx = k, ty): m = ty, ty+8, ... of each tile
    for (int m0 = 0; m0 < N; m0 += 32) {
      for (int r = ty; r < 32; r += 8) {
        // xs[kk][mm] = op(X)[k0+kk][m0+mm]
        if (!T.xdag) {
          const int k = k0 + r, m = m0 + tx;
          xs[r][tx] = (k < N && m < N) ? T.x[(size_t)k * N + m] : make_double2(0.0, 0.0);
        } else {  // op(X)[k][m] = conj(X[m][k]): read row m0+r, columns k0+tx
          const int m = m0 + r, k = k0 + tx;
          double2 v = (k < N && m < N) ? T.x[(size_t)m * N + k] : make_double2(0.0, 0.0);
          xs[tx][r] = make_double2(v.x, -v.y);
        }
        // ys[mm][kk] = op(Y)[m0+mm][k0+kk]
        if (!T.ydag) {
          const int m = m0 + r, k = k0 + tx;
          ys[r][tx] = (k < N && m < N) ? T.y[(size_t)m * N + k] : make_double2(0.0, 0.0);
        } else {  // op(Y)[m][k] = conj(Y[k][m]): read row k0+r, columns m0+tx
          const int k = k0 + r, m = m0 + tx;
          double2 v = (k < N && m < N) ? T.y[(size_t)k * N + m] : make_double2(0.0, 0.0);
          ys[tx][r] = make_double2(v.x, -v.y);
        }
      }
      __syncthreads();
      // only the tile's valid m (the padding beyond N would still cost the FP64 pipe)
      const int mlim = min(32, N - m0);
      for (int mm = ty; mm < mlim; mm += 8) cmac(acc, xs[tx][mm], ys[mm][tx]);
      __syncthreads();
    }
    part[ty][tx] = acc;
    __syncthreads();
    if (ty == 0) {
      double2 d = make_double2(0.0, 0.0);
      for (int q = 0; q < 8; q++) {
        d.x += part[q][tx].x;
        d.y += part[q][tx].y;
      }
      const int k = k0 + tx;
      if (T.out >= 0 && k < N) {
        const double2 w = diag_weight(T);
        buf[(size_t)T.out * N + k] = w.x * d.x - w.y * d.y;
      }
      tot[tx] = k < N ? d : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (T.vout >= 0 && threadIdx.x == 0) {
      for (int q = 0; q < 32; q++) {
        vsum.x += tot[q].x;
        vsum.y += tot[q].y;
      }
    }
    __syncthreads();
  }
  if (T.vout >= 0 && threadIdx.x == 0) vals[T.vout] = vsum;
}

// grad[k] += (sum_t buf[t][k]) / f[k], summed in a fixed order.
__global__ void __launch_bounds__(256) grad_reduce_kernel(const double* __restrict__ buf, int ntask, int N,
                                                          const double* __restrict__ f, double* __restrict__ grad) {
  const int k = blockIdx.x;
  double s = 0.0;
  for (int t = threadIdx.x; t < ntask; t += 256) s += buf[(size_t)t * N + k];
  s = block_sum_256(s);
  if (threadIdx.x == 0) grad[k] += s / f[k];
}

int launch_grad_reduce(const double* buf, int nrow, int N, const double* f, double* grad, cudaStream_t s) {
  TimedLaunch tl(s, "grad_reduce");
  grad_reduce_kernel<<<N, 256, 0, s>>>(buf, nrow, N, f, grad);
  CTR_CUDA(cudaGetLastError());
  return CTR_OK;
}

// Diagonal reductions of a task list, then grad += (sum of their rows) / f where the
// list has gradient rows (nrow > 0).
int launch_diag(const std::vector<DiagTask>& tasks, int nrow, int N, const double* f, double2* vals, double* grad,
                cudaStream_t s) {
  if (tasks.empty()) return CTR_OK;
  void *ddt, *dbuf = nullptr;
  CTR_TRY(upload(WS_ROWTASKS, tasks.data(), tasks.size() * sizeof(DiagTask), &ddt, s));
  if (nrow > 0) CTR_TRY(workspace(WS_ROWS).get((size_t)nrow * N * sizeof(double), &dbuf));
  {
    TimedLaunch tl(s, "diag_reduce");
    if (N <= 128) {
      int P = 1;
      for (int q : {2, 3, 4, 6, 12})
        if (q * N <= DIAG_TPB) P = q;
      const size_t smem = ((size_t)N * (DK + 1) + (size_t)DK * (N + 1)) * sizeof(double2);
      static_assert((128 * (DK + 1) + DK * 129) * sizeof(double2) <= 56 * 1024, "shared memory of diag_small_kernel");
      CTR_CUDA(cudaFuncSetAttribute(diag_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 56 * 1024));
      diag_small_kernel<<<(unsigned)tasks.size(), DIAG_TPB, smem, s>>>((const DiagTask*)ddt, N, P, (double*)dbuf, vals);
    } else {
      diag_reduce_kernel<<<(unsigned)tasks.size(), 256, 0, s>>>((const DiagTask*)ddt, N, (double*)dbuf, vals);
    }
    CTR_CUDA(cudaGetLastError());
  }
  if (nrow > 0) CTR_TRY(launch_grad_reduce((const double*)dbuf, nrow, N, f, grad, s));
  return CTR_OK;
}

// Sums over pairs of blocks.  A group's elementwise products
//   S[k][m] = sum_j i^u_j X_j[k][m] Y_j[m][k]   (X_j, Y_j conjugated where bit 2 of u_j is set)
// hold all that its traces' value and gradient need: their sum over the first nval
// terms is the value, and the row and column sums of Re(w S) are the terms of
// f_k d/df_k at the two indices the traces are cut at.  So a term takes 4 FMAs an
// element, where a diagonal of X Y and one of Y X took 8 in two passes over its
// blocks.  One CTA a group and tile of S, which stays in registers over the terms;
// the tile's edge is Nev / ceil(Nev / 32), so that no lane of the FP64 pipe, the
// bound, works on padding.  Nev = 100, rho at 512 pairs and pi pi at 64: 60 000 terms
// in 4.7 ms (4.1 ms of FMAs) where the diagonals took 10.9.
struct PairTerm {
  const double2* x;
  const double2* y;
  int unit;  // u_j
  int pad;
};
struct PairGroup {
  int first, n;     // terms
  int nval;         // terms of the value, 0: none wanted
  int row;          // first gradient row (2 nt rows), -1: none wanted
  double scale;     // of S
  double wre, wim;  // weight, times *wp where wp is set
  const double2* wp;
};
__device__ __forceinline__ double flip_sign(double v, int mask) {
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

constexpr int PS_T = 32, PS_J = 4, PS_TPB = PS_T * PS_T / PS_J;

__global__ void __launch_bounds__(PS_TPB) pair_sums_kernel(const PairGroup* __restrict__ groups,
                                                           const PairTerm* __restrict__ terms, int N, int T, int nt,
                                                           double* __restrict__ buf, double2* __restrict__ part) {
  __shared__ double2 ys[2][PS_T * (PS_T + 1)];  // Y's tile, transposed
  __shared__ double red[PS_TPB / 32][2];
  const PairGroup G = groups[blockIdx.x / (nt * nt)];
  const int tile = blockIdx.x % (nt * nt), tk = tile / nt, tm = tile % nt, k0 = tk * T, m0 = tm * T;
  const int nk = min(T, N - k0), nm = min(T, N - m0);
  // element e of the tile: row e / T, column e % T of X's and of Y's tile
  int xo[PS_J], yo[PS_J], rd[PS_J], wr[PS_J];
#pragma unroll
  for (int j = 0; j < PS_J; j++) {
    const int e = threadIdx.x + j * (int)blockDim.x, r = e / T, q = e - r * T;
    xo[j] = r < nk && q < nm ? (k0 + r) * N + m0 + q : -1;
    yo[j] = r < nm && q < nk ? (m0 + r) * N + k0 + q : -1;
    rd[j] = r < T ? r * (T + 1) + q : 0;
    wr[j] = r < T ? q * (T + 1) + r : -1;
  }
  double2 x[PS_J], y[PS_J], S[PS_J];
  double2 v = make_double2(0.0, 0.0);
  int unit = 0;
#pragma unroll
  for (int j = 0; j < PS_J; j++) S[j] = make_double2(0.0, 0.0);
  auto load = [&](int i) {
    const PairTerm P = terms[G.first + i];
    unit = P.unit;
#pragma unroll
    for (int j = 0; j < PS_J; j++) {
      x[j] = xo[j] >= 0 ? P.x[xo[j]] : make_double2(0.0, 0.0);
      y[j] = yo[j] >= 0 ? P.y[yo[j]] : make_double2(0.0, 0.0);
    }
  };
  load(0);
  for (int i = 0; i < G.n; i++) {
    double2* const Y = ys[i & 1];
    double2 a[PS_J];
    // a = i^u x, signs as integer operations (a negation of a double takes the FP64 pipe)
    const int conj = unit & 4 ? 1 << 31 : 0, neg = unit & 2 ? 1 << 31 : 0;
    const bool swap = unit & 1;
    const int sx = swap ? neg ^ conj ^ (1 << 31) : neg, sy = swap ? neg : neg ^ conj;
#pragma unroll
    for (int j = 0; j < PS_J; j++) {
      if (wr[j] >= 0) Y[wr[j]] = make_double2(y[j].x, flip_sign(y[j].y, conj));
      a[j].x = flip_sign(swap ? x[j].y : x[j].x, sx);
      a[j].y = flip_sign(swap ? x[j].x : x[j].y, sy);
    }
    if (i + 1 < G.n) load(i + 1);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PS_J; j++) cmac(S[j], a[j], Y[rd[j]]);
    if (i + 1 == G.nval) {
#pragma unroll
      for (int j = 0; j < PS_J; j++) {
        v.x += S[j].x;
        v.y += S[j].y;
      }
    }
  }
  if (G.nval > 0) {
    for (int o = 16; o; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][0] = v.x, red[threadIdx.x >> 5][1] = v.y;
  }
  __syncthreads();
  if (G.nval > 0 && threadIdx.x == 0) {
    double2 z = make_double2(red[0][0], red[0][1]);
    for (int w = 1; w < (int)blockDim.x / 32; w++) {
      z.x += red[w][0];
      z.y += red[w][1];
    }
    part[blockIdx.x] = make_double2(G.scale * z.x, G.scale * z.y);
  }
  if (G.row < 0) return;
  double2 w = make_double2(G.scale * G.wre, G.scale * G.wim);
  if (G.wp) w = cmul(w, *G.wp);
  double* const R = (double*)ys[0];
#pragma unroll
  for (int j = 0; j < PS_J; j++)
    if (wr[j] >= 0) R[rd[j]] = w.x * S[j].x - w.y * S[j].y;
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * T; t += blockDim.x) {
    double s = 0.0;
    if (t < T) {
      if (t >= nk) continue;
      for (int q = 0; q < nm; q++) s += R[t * (T + 1) + q];
      buf[(size_t)(G.row + tm) * N + k0 + t] = s;
    } else {
      if (t - T >= nm) continue;
      for (int r = 0; r < nk; r++) s += R[r * (T + 1) + t - T];
      buf[(size_t)(G.row + nt + tk) * N + m0 + t - T] = s;
    }
  }
}

// out[ent[g]] = sum of the group's tiles' parts.
__global__ void pair_value_kernel(const double2* __restrict__ part, int ntile, const int* __restrict__ ent, int n,
                                  double2* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  double2 z = part[(size_t)g * ntile];
  for (int t = 1; t < ntile; t++) {
    z.x += part[(size_t)g * ntile + t].x;
    z.y += part[(size_t)g * ntile + t].y;
  }
  out[ent[g]] = z;
}

// Power u of i with c = |c| i^u, -1 where there is none.
int unit_of(float re, float im) {
  if (im == 0.f) return re > 0.f ? 0 : 2;
  if (re == 0.f) return im > 0.f ? 1 : 3;
  return -1;
}

// A list of groups; run: values to out[ent[g]] (one entry a group, where ent is not
// empty) and grad += (gradient terms) / f where grad is set.
struct PairList {
  std::vector<PairGroup> g;
  std::vector<PairTerm> t;
  std::vector<int> ent;
  void begin(double2 w, const double2* wp = nullptr, double scale = 1.0) {
    g.push_back({(int)t.size(), 0, 0, -1, scale, w.x, w.y, wp});
  }
  void term(const double2* x, const double2* y, int unit = 0) {
    t.push_back({x, y, unit, 0});
    g.back().n++;
  }
  int run(int N, const double* f, double2* out, double* grad, cudaStream_t s) {
    if (g.empty()) return CTR_OK;
    const int nt = (N + PS_T - 1) / PS_T, T = (N + nt - 1) / nt;
    const long long grid = (long long)g.size() * nt * nt;
    if (grid > 0x7fffffffLL) return fail(CTR_ERR_ARG, "profile gradient: too many groups (%zu)", g.size());
    if (grad)
      for (size_t k = 0; k < g.size(); k++) g[k].row = (int)k * 2 * nt;
    void *d[3], *dbuf = nullptr, *dpart = nullptr;
    CTR_TRY(upload_group(WS_ROWTASKS,
                         {{g.data(), g.size() * sizeof(PairGroup)},
                          {t.data(), t.size() * sizeof(PairTerm)},
                          {ent.data(), ent.size() * sizeof(int)}},
                         d, s));
    const int nrow = grad ? (int)g.size() * 2 * nt : 0;
    if (grad) CTR_TRY(workspace(WS_ROWS).get((size_t)nrow * N * sizeof(double), &dbuf));
    if (!ent.empty()) CTR_TRY(workspace(WS_ROWABS).get((size_t)grid * sizeof(double2), &dpart));
    {
      TimedLaunch tl(s, "pair_sums");
      const int tpb = std::max(32, (T * T + PS_J * 32 - 1) / (PS_J * 32) * 32);
      pair_sums_kernel<<<(unsigned)grid, tpb, 0, s>>>((const PairGroup*)d[0], (const PairTerm*)d[1], N, T, nt,
                                                      (double*)dbuf, (double2*)dpart);
      CTR_CUDA(cudaGetLastError());
    }
    if (!ent.empty()) {
      TimedLaunch tl(s, "pair_value");
      const int n = (int)ent.size();
      pair_value_kernel<<<(n + 63) / 64, 64, 0, s>>>((const double2*)dpart, nt * nt, (const int*)d[2], n, out);
      CTR_CUDA(cudaGetLastError());
    }
    if (grad) CTR_TRY(launch_grad_reduce((const double*)dbuf, nrow, N, f, grad, s));
    return CTR_OK;
  }
};

// ------------------------------------------------------------- chain program
inline int64_t factor_key(const ctr_factor& F) {
  return ((((((int64_t)F.kind * 2 + (F.dag ? 1 : 0)) * 8192 + F.a) * 8192 + F.b) * 4 + F.s1) * 4 + F.s2);
}

struct Opnd {
  const double2* p;
  int dag;
};

class ChainProgram {
 public:
  ChainProgram(int N, int Nt, int nphi, const double2* prop, const double2* phis, int engine)
      : N_(N), Nt_(Nt), nphi_(nphi), engine_(engine), prop_(prop), phis_(phis) {}

  int check_factor(const ctr_factor& F) const {
    if (F.kind == CTR_FACTOR_TAU) {
      if (F.a < 0 || F.a >= Nt_ || F.b < 0 || F.b >= Nt_ || F.s1 < 0 || F.s1 > 3 || F.s2 < 0 || F.s2 > 3)
        return fail(CTR_ERR_ARG, "chain factor: perambulator block out of range");
    } else if (F.kind == CTR_FACTOR_PHI) {
      if (F.a < 0 || F.a >= Nt_ || F.b < 0 || F.b >= nphi_)
        return fail(CTR_ERR_ARG, "chain factor: elemental out of range");
    } else {
      return fail(CTR_ERR_ARG, "chain factor: unknown kind %d", F.kind);
    }
    return CTR_OK;
  }

  Opnd leaf(const ctr_factor& F) const {
    const size_t N2 = (size_t)N_ * N_;
    if (F.kind == CTR_FACTOR_TAU)
      return Opnd{prop_ + (((size_t)F.a * Nt_ + F.b) * 16 + F.s1 * 4 + F.s2) * N2, F.dag ? 1 : 0};
    return Opnd{phis_ + ((size_t)F.a * nphi_ + F.b) * N2, F.dag ? 1 : 0};
  }

  // Adds one chain; returns the number of new GEMM nodes it needed.
  int add(const ctr_factor* F, int n, double2 w, int value_slot, bool grad) {
    Chain c;
    c.f.assign(F, F + n);
    c.w = w;
    c.value_slot = value_slot;
    c.grad = grad;
    const int before = (int)nodes_.size();
    // prefixes P_1 .. P_{n-1} (P_1 is the leaf F_1); operand ids: >= 0 node, < 0 leaf index in chain
    c.pre.assign(n, -1);
    int64_t cur = -(1 + factor_key(F[0]));
    c.pre[0] = -1;
    for (int j = 1; j < n - 1; j++) {
      cur = node(cur, -(1 + factor_key(F[j])), j + 1, F, j, true, c.pre[j - 1]);
      c.pre[j] = (int)cur;
    }
    // suffixes S_n .. S_2 (S_n is the leaf F_n); a chain without gradient needs none
    c.suf.assign(n + 1, -1);
    cur = -(1 + factor_key(F[n - 1]));
    for (int j = n - 2; j >= 1 && grad; j--) {
      cur = node(-(1 + factor_key(F[j])), cur, n - j, F, j, false, c.suf[j + 1]);
      c.suf[j] = (int)cur;
    }
    chains_.push_back(std::move(c));
    return (int)nodes_.size() - before;
  }

  size_t nodes() const { return nodes_.size(); }

  void clear() {
    nodes_.clear();
    chains_.clear();
    pre_map_.clear();
    suf_map_.clear();
  }

  // Executes the program: GEMM levels, diagonal reductions, gradient sum.
  int run(const double* f, double2* values, double* grad, cudaStream_t s);

 private:
  struct Node {
    int depth;
    int a_node, b_node;  // >= 0: operand is node; -1: leaf
    Opnd a_leaf, b_leaf;
  };
  struct Chain {
    std::vector<ctr_factor> f;
    std::vector<int> pre, suf;  // node ids (-1 = leaf)
    double2 w;
    int value_slot;
    bool grad;
  };

  // prefix node: parent (node id >= 0 or leaf key < 0) x factor F[j]
  // suffix node: factor F[j] x child
  int64_t node(int64_t left, int64_t right, int depth, const ctr_factor* F, int j, bool prefix, int other_node) {
    auto& map = prefix ? pre_map_ : suf_map_;
    const auto key = std::make_pair(left, right);
    auto it = map.find(key);
    if (it != map.end()) return it->second;
    Node nd;
    nd.depth = depth;
    if (prefix) {
      nd.a_node = other_node;  // parent node (or -1 if P_1 is a leaf)
      nd.a_leaf = leaf(F[0]);
      nd.b_node = -1;
      nd.b_leaf = leaf(F[j]);
    } else {
      nd.a_node = -1;
      nd.a_leaf = leaf(F[j]);
      nd.b_node = other_node;  // child node (or -1 if S_{j+1} is the leaf F_n)
      nd.b_leaf = leaf(F[j + 1]);
    }
    const int id = (int)nodes_.size();
    nodes_.push_back(nd);
    map.emplace(key, id);
    return id;
  }

  int N_, Nt_, nphi_, engine_;
  const double2* prop_;
  const double2* phis_;
  std::vector<Node> nodes_;
  std::vector<Chain> chains_;
  std::map<std::pair<int64_t, int64_t>, int> pre_map_, suf_map_;
};

int ChainProgram::run(const double* f, double2* values, double* grad, cudaStream_t s) {
  if (chains_.empty()) return CTR_OK;
  const size_t N2 = (size_t)N_ * N_;
  void* nodemem = nullptr;
  CTR_TRY(workspace(WS_SCRATCH).get(std::max<size_t>(1, nodes_.size()) * N2 * sizeof(double2), &nodemem));
  double2* nb = (double2*)nodemem;
  auto opnd = [&](int node_id, const Opnd& lf) { return node_id >= 0 ? Opnd{nb + (size_t)node_id * N2, 0} : lf; };

  // GEMM levels: nodes of equal depth are independent; one upload, one launch per depth
  int maxd = 0;
  for (const Node& nd : nodes_) maxd = std::max(maxd, nd.depth);
  std::vector<ZTask> tasks;
  std::vector<size_t> level_off(maxd + 2, 0);
  for (int d = 2; d <= maxd; d++) {
    level_off[d] = tasks.size();
    for (size_t i = 0; i < nodes_.size(); i++) {
      const Node& nd = nodes_[i];
      if (nd.depth != d) continue;
      const Opnd a = opnd(nd.a_node, nd.a_leaf), b = opnd(nd.b_node, nd.b_leaf);
      ZTask t;
      std::memset(&t, 0, sizeof(t));
      t.A[0] = a.p;
      t.B[0] = b.p;
      t.C = nb + i * N2;
      t.wre[0] = 1.f;
      t.nterm = 1;
      t.flags = (a.dag ? 1 : 0) | (b.dag ? 16 : 0);
      tasks.push_back(t);
    }
  }
  level_off[maxd + 1] = tasks.size();
  if (!tasks.empty() && engine_ == CTR_ENGINE_SPLIT) {
    for (int d = 2; d <= maxd; d++) {
      const size_t n0 = level_off[d], n1 = level_off[d + 1];
      if (n1 > n0) CTR_TRY(zgemm_split_tasks(N_, tasks.data() + n0, (int)(n1 - n0), s));
    }
  } else if (!tasks.empty()) {
    void* dt;
    CTR_TRY(upload(WS_GEMM_A, tasks.data(), tasks.size() * sizeof(ZTask), &dt, s));
    for (int d = 2; d <= maxd; d++) {
      const size_t n0 = level_off[d], n1 = level_off[d + 1];
      if (n1 > n0) CTR_TRY(launch_zgemm_f64((const ZTask*)dt + n0, (int)(n1 - n0), N_, s, tasks.data() + n0));
    }
  }

  // diagonal reductions (gradient) and traces (values)
  std::vector<DiagTask> dtasks;
  int ngrad = 0;
  for (const Chain& c : chains_) {
    const int n = (int)c.f.size();
    auto P = [&](int j) { return opnd(c.pre[j - 1], leaf(c.f[0])); };  // P_j, j = 1..n-1
    auto S = [&](int j) { return opnd(c.suf[j - 1], leaf(c.f[n - 1])); };  // S_j, j = 2..n
    auto F = [&](int j) { return leaf(c.f[j - 1]); };
    auto push = [&](Opnd x, Opnd y, int out, int vout) {
      DiagTask t;
      std::memset(&t, 0, sizeof(t));
      t.x = x.p;
      t.y = y.p;
      t.xdag = x.dag;
      t.ydag = y.dag;
      t.wre = c.w.x;
      t.wim = c.w.y;
      t.out = out;
      t.vout = vout;
      dtasks.push_back(t);
    };
    if (c.value_slot >= 0) push(P(n - 1), F(n), -1, c.value_slot);  // Tr = sum diag(P_{n-1} F_n)
    if (!c.grad) continue;
    for (int j = 1; j <= n; j++) {
      if (c.f[j - 1].kind != CTR_FACTOR_PHI) continue;
      // left D of F_j: diag(S_j P_{j-1}); j = 1: diag(F_1 S_2)
      if (j == 1) push(F(1), S(2), ngrad++, -1);
      else push(S(j), P(j - 1), ngrad++, -1);
      // right D of F_j: diag(S_{j+1} P_j); j = n: diag(P_{n-1} F_n)
      if (j == n) push(P(n - 1), F(n), ngrad++, -1);
      else push(S(j + 1), P(j), ngrad++, -1);
    }
  }
  return launch_diag(dtasks, ngrad, N_, f, values, grad, s);
}

// Runs chains through programs of bounded size (node storage <= budget).
class ChainRunner {
 public:
  ChainRunner(int N, int Nt, int nphi, const double2* prop, const double2* phis, const double* f, double2* values,
              double* grad, cudaStream_t s, int engine = CTR_ENGINE_FP64)
      : prog_(N, Nt, nphi, prop, phis, engine), f_(f), values_(values), grad_(grad), s_(s) {
    const size_t budget = (size_t)3 << 30;
    max_nodes_ = std::max<size_t>(64, budget / ((size_t)N * N * sizeof(double2)));
  }
  int check(const ctr_factor& F) const { return prog_.check_factor(F); }
  // Chains of one group (e.g. one (t_sink, t_src) pair) are added together.
  int add(const ctr_factor* F, int n, double2 w, int value_slot, bool grad) {
    prog_.add(F, n, w, value_slot, grad);
    return CTR_OK;
  }
  int end_group() {
    if (prog_.nodes() >= max_nodes_ / 2) return flush();
    return CTR_OK;
  }
  int flush() {
    CTR_TRY(prog_.run(f_, values_, grad_, s_));
    prog_.clear();
    return CTR_OK;
  }

 private:
  ChainProgram prog_;
  const double* f_;
  double2* values_;
  double* grad_;
  cudaStream_t s_;
  size_t max_nodes_;
};

// Scaled elemental copies diag(f) Phi diag(f) in a workspace slot.
int profiled(int N, long long nmat, const double* phi, const double* f, int slot, double2** out, cudaStream_t s) {
  void* p;
  CTR_TRY(workspace(slot).get((size_t)nmat * N * N * sizeof(double2), &p));
  TimedLaunch tl(s, "apply_profile");
  apply_profile_kernel<<<1024, 256, 0, s>>>((const double2*)phi, (double2*)p, f, N, nmat);
  CTR_CUDA(cudaGetLastError());
  *out = (double2*)p;
  return CTR_OK;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// A gradient's correlators, of which the caller's array need only hold doubles: the kernels
// write p, 16-byte aligned, and close() copies it to the array where it is not.
struct CorrOut {
  double* to;
  size_t n;
  double2* p = nullptr;
  CorrOut(double* corr, size_t entries) : to(corr), n(entries) {}
  int open() {
    p = (double2*)to;
    void* m;
    if (aligned16(to)) return CTR_OK;
    CTR_TRY(workspace(WS_ADJ_CORR).get(n * sizeof(double2), &m));
    p = (double2*)m;
    return CTR_OK;
  }
  int close(cudaStream_t s) const {
    if (p != (double2*)to) CTR_CUDA(cudaMemcpyAsync(to, p, n * sizeof(double2), cudaMemcpyDeviceToDevice, s));
    return CTR_OK;
  }
};

int check_f(int N, const double* f, cudaStream_t s) {
  std::vector<double> h(N);
  CTR_CUDA(cudaMemcpyAsync(h.data(), f, N * sizeof(double), cudaMemcpyDeviceToHost, s));
  CTR_CUDA(cudaStreamSynchronize(s));
  for (int k = 0; k < N; k++)
    if (!(h[k] != 0.0) || !std::isfinite(h[k])) return fail(CTR_ERR_ARG, "profile f[%d] = %g must be finite and nonzero", k, h[k]);
  return CTR_OK;
}

int check_engine(int engine, int nev) {
  if (engine != CTR_ENGINE_FP64 && engine != CTR_ENGINE_SPLIT) return fail(CTR_ERR_ARG, "unknown engine %d", engine);
  return CTR_OK;
}

// ------------------------------------------------------- rho and pi pi gradients
// Products of a batch in one workspace buffer.
struct Arena {
  double2* base = nullptr;
  size_t N2 = 0, used = 0, cap = 0;
  double2* take(size_t nblk) {
    double2* p = base + used;
    used += nblk * N2;
    return p;
  }
};

// Pairs (tf * Nt + ti) with a nonzero weight, those of one source time together.
std::vector<int> weighted_pairs(int Nt, int nout, const double2* w) {
  std::vector<int> p;
  for (int ti = 0; ti < Nt; ti++)
    for (int tf = 0; tf < Nt; tf++) {
      const double2* wp = w + ((size_t)tf * Nt + ti) * nout;
      for (int k = 0; k < nout; k++)
        if (wp[k].x != 0.0 || wp[k].y != 0.0) {
          p.push_back(tf * Nt + ti);
          break;
        }
    }
  return p;
}

// Host tables of a batch.
constexpr size_t TABLE_BUDGET = (size_t)64 << 20;

// rho (lib/calculate_rho_core.h): a spin row is coef * t, t = Tr[A_cd Bt_ab] with
// A = tau_cd Phi_L(ti) and Bt = tau_ab^dag Phi_R(tf)^dag, so f_k d/df_k of t is
// diag(Bt A) at Phi_L's right index and diag(A Bt) at Phi_R's left one.  Cut at the
// other two indices, conj(t) = Tr[At_ab Bs_cd] with At = tau_ab Phi_L(ti)^dag and Bs =
// tau_cd^dag Phi_R(tf): diag(Bs At) is Phi_L's left index, diag(At Bs) Phi_R's right one.
// Per pair and operator that is 64 block products, whatever the number of rows.
int rho_vjp(const Ctx& c, const double2* prop, const double2* phis, const double* f, const double2* w, double2* corr,
            double* grad) {
  const int N = c.N, Nt = c.Nt;
  const size_t N2 = c.N2, blk16 = 16 * N2;
  if (corr) CTR_CUDA(cudaMemsetAsync(corr, 0, (size_t)Nt * Nt * 48 * sizeof(double2), c.s));
  const std::vector<int> pairs = weighted_pairs(Nt, 48, w);
  if (pairs.empty()) return CTR_OK;
  const Tables& T = tables();
  // operators used at the source (L) and at the sink (R)
  std::vector<int> Ls, Rs, il(5, -1), ir(5, -1);
  for (int p : pairs)
    for (int o = 0; o < 48; o++) {
      const double2 wo = w[(size_t)p * 48 + o];
      if (wo.x == 0.0 && wo.y == 0.0) continue;
      for (int is = 0; is < 16; is++) {
        const int l = T.rho_lprp[o * 16 + is][0], r = T.rho_lprp[o * 16 + is][1];
        if (il[l] < 0) il[l] = (int)Ls.size(), Ls.push_back(l);
        if (ir[r] < 0) ir[r] = (int)Rs.size(), Rs.push_back(r);
      }
    }
  const int nL = (int)Ls.size(), nR = (int)Rs.size(), kinds = grad ? 2 : 1;
  const size_t per_pair = 16 * (size_t)kinds * (nL + nR) * N2 * sizeof(double2);
  // a pair's terms, at most 48 outputs of them; a batch's tables pass through a pinned
  // staging buffer, so they are bounded as well as its blocks
  const size_t table = 48 * (sizeof(PairGroup) + 16 * (size_t)kinds * sizeof(PairTerm));
  const int batch = (int)std::max<size_t>(1, std::min({pairs.size(), CHAIN_BUDGET / per_pair, TABLE_BUDGET / table}));
  for (const PairBatch& pb : pair_batches(prop, blk16, Nt, 0, Nt, batch, &pairs)) {
    const int np = (int)pb.ent.size();
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get((size_t)np * per_pair, &mem));
    Arena ar;
    ar.base = (double2*)mem;
    ar.N2 = N2;
    // side 0: tau against [Phi_L, Phi_L^dag] per t_src; side 1: tau^dag against [Phi_R^dag, Phi_R] per t_sink
    std::vector<GridTask> g0;
    std::vector<double2*> bs[2];
    for (int side = 0; side < 2; side++) {
      const auto& groups = side ? pb.by_tf : pb.by_ti;
      const std::vector<int>& ops = side ? Rs : Ls;
      const int nr = kinds * (int)ops.size();
      for (const std::vector<int>& mem_i : groups) {
        const int m = (int)mem_i.size(), t = side ? pb.tf[mem_i[0]] : pb.ti[mem_i[0]];
        double2* out = ar.take((size_t)16 * m * nr);
        bs[side].push_back(out);
        for (int r0 = 0; r0 < nr; r0 += 8) {
          GridTask G = make_grid(16 * m, std::min(8, nr - r0), 1, kOne, side, 0);
          for (int pp = 0; pp < m; pp++)
            for (int b = 0; b < 16; b++) G.A[pp * 16 + b] = pb.T[mem_i[pp]] + (size_t)b * N2;
          for (int j = 0; j < G.nb; j++) {
            const int op = (r0 + j) / kinds, dag = ((r0 + j) % kinds) ^ side;
            G.B[j][0] = phis + ((size_t)t * 5 + ops[op]) * N2;
            G.bdag |= dag << (4 * j);
            G.C0[j] = out + (size_t)(r0 + j) * 16 * m * N2;
          }
          g0.push_back(std::move(G));
        }
      }
    }
    auto blk = [&](int side, int i, int op, int kind, int b) {
      const int g = side ? pb.gtf[i] : pb.gti[i], pos = side ? pb.ptf[i] : pb.pti[i];
      const size_t m = side ? pb.by_tf[g].size() : pb.by_ti[g].size();
      return bs[side][g] + (((size_t)(op * kinds + kind) * m + pos) * 16 + b) * N2;
    };
    // an output's 16 rows: its value, and f d/df at Phi_L's right and Phi_R's left index,
    // from the first cut; the other two indices from the second one's conjugates
    PairList pl;
    for (int i = 0; i < np; i++) {
      const int pr = pairs[pb.ent[i]];
      for (int o = 0; o < 48; o++) {
        const double2 wo = w[(size_t)pr * 48 + o];
        if (wo.x == 0.0 && wo.y == 0.0) continue;
        // the rows' coefficients are one magnitude, a power of two, times powers of i
        auto mag = [&](int r) { return std::max(std::fabs(T.rho_coef[r][0]), std::fabs(T.rho_coef[r][1])); };
        pl.begin(wo, nullptr, mag(o * 16));
        for (int kind = 0; kind < kinds; kind++)
          for (int is = 0; is < 16; is++) {
            const int r = o * 16 + is, u = unit_of(T.rho_coef[r][0], T.rho_coef[r][1]);
            if (u < 0 || mag(r) != mag(o * 16)) return fail(CTR_ERR_ARG, "rho row %d: unexpected coefficient", r);
            const int16_t* sp = T.rho_spin[r];
            const int cd = sp[2] * 4 + sp[3], ab = sp[0] * 4 + sp[1], l = il[T.rho_lprp[r][0]], q = ir[T.rho_lprp[r][1]];
            pl.term(blk(0, i, l, kind, kind ? ab : cd), blk(1, i, q, kind, kind ? cd : ab), u + 4 * kind);
          }
        if (corr) {
          pl.g.back().nval = 16;
          pl.ent.push_back(pr * 48 + o);
        }
      }
    }
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(pl.run(N, f, corr, grad, c.s));
  }
  return CTR_OK;
}

// out = sum_k w_k in_k (added to out where add is set), one CTA column per block.
struct CombTask {
  double2* out;
  int first, n, add, pad;
};
struct CombIn {
  const double2* in;
  double2 w;
};
__global__ void __launch_bounds__(256) combine_blocks_kernel(const CombTask* __restrict__ tasks,
                                                             const CombIn* __restrict__ in, int n2) {
  const CombTask T = tasks[blockIdx.x];
  for (int e = threadIdx.x; e < n2; e += 256) {
    double2 v = T.add ? T.out[e] : make_double2(0.0, 0.0);
    for (int k = 0; k < T.n; k++) cmac(v, in[T.first + k].w, in[T.first + k].in[e]);
    T.out[e] = v;
  }
}

struct CombList {
  std::vector<CombTask> t;
  std::vector<CombIn> in;
  void begin(double2* out, bool add) { t.push_back(CombTask{out, (int)in.size(), 0, add ? 1 : 0, 0}); }
  void term(const double2* x, double2 w) {
    in.push_back(CombIn{x, w});
    t.back().n++;
  }
  int run(int n2, cudaStream_t s) {
    if (t.empty()) return CTR_OK;
    void* d[2];
    CTR_TRY(upload_group(WS_TASKS2, {{t.data(), t.size() * sizeof(CombTask)}, {in.data(), in.size() * sizeof(CombIn)}},
                         d, s));
    TimedLaunch tl(s, "combine_blocks");
    combine_blocks_kernel<<<(unsigned)t.size(), 256, 0, s>>>((const CombTask*)d[0], (const CombIn*)d[1], n2);
    CTR_CUDA(cudaGetLastError());
    return CTR_OK;
  }
};

// Per pair: vals [64] = 16 each of square, double triangle, horizontal double triangle
// and 4 x 4 of the twin traces (P4, P1), (P3, P2), (P3, P1), (P4, P2); corr [5] the
// weighted slots; twin weights wk [4]: star = t0 t1, fish = t2 t3, so d(star) = t1 dt0 + t0 dt1.
__global__ void pipi_vjp_combine_kernel(const double2* __restrict__ vals, const int* __restrict__ ent,
                                        const double2* __restrict__ wsf, int npair, double wsq, double wdt, double wst,
                                        double wfi, double wdh, double2* __restrict__ corr, double2* __restrict__ wk) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  const double2* v = vals + (size_t)p * 64;
  double2 a[3], t[4];
  for (int g = 0; g < 3; g++) {
    a[g] = make_double2(0.0, 0.0);
    for (int b = 0; b < 16; b++) {
      // the 4x4 block matrices carry gamma_5 on the first index of square and double triangle
      const double sg = g < 2 && b >= 8 ? -1.0 : 1.0;
      a[g].x += sg * v[g * 16 + b].x;
      a[g].y += sg * v[g * 16 + b].y;
    }
  }
  for (int k = 0; k < 4; k++) {
    t[k] = make_double2(0.0, 0.0);
    for (int b = 0; b < 4; b++) {
      t[k].x += v[48 + k * 4 + b].x;
      t[k].y += v[48 + k * 4 + b].y;
    }
  }
  if (corr) {
    const double2 st = cmul(t[0], t[1]), fi = cmul(t[2], t[3]);
    double2* o = corr + (size_t)ent[p] * 5;
    o[0] = make_double2(wsq * a[0].x, wsq * a[0].y);
    o[1] = make_double2(wdt * a[1].x, wdt * a[1].y);
    o[2] = make_double2(wst * st.x, wst * st.y);
    o[3] = make_double2(wfi * fi.x, wfi * fi.y);
    o[4] = make_double2(wdh * a[2].x, wdh * a[2].y);
  }
  const double2 ws = wsf[2 * p], wf = wsf[2 * p + 1];
  wk[4 * p] = cmul(ws, t[1]);
  wk[4 * p + 1] = cmul(ws, t[0]);
  wk[4 * p + 2] = cmul(wf, t[3]);
  wk[4 * p + 3] = cmul(wf, t[2]);
}

// pi pi.  Per pair, T = tau(tf, ti) as a 4x4 block matrix, W = T^dag L:
//   square = Tr[Rsq J], double triangle = Tr[Rdt J],  J = W G T G,
//   w_sq square + w_dt double triangle = Tr[L K],     K = G T G (w_sq Rsq + w_dt Rdt) T^dag,
// so J (weighted, summed per t_src) is the co-factor of R = Phi tau(ti,ti) Phi and K
// (summed per t_sink) that of L: what remains is a product of two elementals and two
// block matrices per time slice.  The horizontal double triangle is Tr[P3 Pm1 P4 Pm2],
// Pm_q = T P_q T^dag, cut at P3 and P4 as (P3 Pm1)(P4 Pm2) and (Pm1 P4)(Pm2 P3), and
// Tr[P1 N1], N1 = sum T^dag (P4 Pm2 P3) T at P1.  The star / fish twins are
// Tr[P_x sum_c Pm_cc(y)] = Tr[P_y sum tau^dag P_x tau].  About 700 block products a pair
// where one chain per spin row took 6 000 and 14 000 diagonals.
int pipi_vjp(const Ctx& c, int iso, const double2* prop, const std::vector<Elem>& el, const int32_t* q, const double* f,
             const double2* w, double2* corr, double* grad) {
  const int N = c.N, Nt = c.Nt;
  const size_t N2 = c.N2, blk16 = 16 * N2;
  if (corr) CTR_CUDA(cudaMemsetAsync(corr, 0, (size_t)Nt * Nt * 5 * sizeof(double2), c.s));
  const std::vector<int> pairs = weighted_pairs(Nt, 5, w);
  if (pairs.empty()) return CTR_OK;
  // isospin weights of the correlator slots (lib/contract_kernels_pipi.cu:288-303, :463-478)
  const double wsq = iso == 1 ? -2.0 : -1.0 / 3.0, wdt = iso == 1 ? 2.0 : -1.0 / 3.0;
  const double wst = iso == 1 ? -1.0 : 1.0, wfi = 1.0, wdh = iso == 1 ? 0.0 : -5.0 / 3.0;
  const bool g = grad != nullptr, hor = iso == 0;
  auto P = [&](int k, int t) { return el[q[k]].p + (size_t)t * el[q[k]].stride; };  // k = 0..3: P1..P4
  enum { P1 = 0, P2 = 1, P3 = 2, P4 = 3 };
  Combos cb(Nt);
  const int cL = cb.use(q[P3], q[P4]), cSq = cb.use(q[P2], q[P1]), cDt = cb.use(q[P1], q[P2]);
  std::vector<char> on_tf(Nt, 0), on_ti(Nt, 0);
  for (int p : pairs) {
    on_tf[p / Nt] = on_ti[p % Nt] = 1;
    cb.need[cL][p / Nt] = cb.need[cSq][p % Nt] = cb.need[cDt][p % Nt] = 1;
  }
  std::vector<const double2*> M;
  // tau(t, t) of the full perambulator
  CTR_TRY(per_t_products(c, prop, (size_t)(Nt + 1) * blk16, el, WS_RPHI, cb.list, cb.need, 16 * (4 * (size_t)Nt + 4), M));
  // The co-factors K and J carry the weights through block products, whose operands flush
  // to zero below 2^-1000: they take the weights relative to a power of two.
  double wmax = 0.0;
  for (int p : pairs)
    for (int k = 0; k < 2; k++)
      wmax = std::max({wmax, std::fabs(w[(size_t)p * 5 + k].x), std::fabs(w[(size_t)p * 5 + k].y)});
  const int wexp = wmax > 0.0 && std::isfinite(wmax) ? std::max(-1000, std::min(1000, std::ilogb(wmax))) : 0;
  const double wdown = std::ldexp(1.0, -wexp), wup = std::ldexp(1.0, wexp);
  // co-factors per time slice: K [tf][16], Jsq, Jdt [ti][16] (block (row, column) of the co-factor)
  double2 *Ks = nullptr, *Js = nullptr, *Jd = nullptr;
  if (g) {
    void* am;
    CTR_TRY(workspace(WS_ADJ_SUM).get(3 * (size_t)Nt * blk16 * sizeof(double2), &am));
    CTR_CUDA(cudaMemsetAsync(am, 0, 3 * (size_t)Nt * blk16 * sizeof(double2), c.s));
    Ks = (double2*)am;
    Js = Ks + (size_t)Nt * blk16;
    Jd = Js + (size_t)Nt * blk16;
  }
  const size_t blocks = 32 + 32 + (hor ? 32 : 8)          // W, J; V; Pm
                        + (hor ? 32 : 0)                  // X1, X2
                        + (g ? 48 + 32 + 8 : 0)           // Rw, S, K; U; O
                        + (g && hor ? 32 + 32 + 32 + 8 : 0);  // Y; Z; Q; N
  const size_t per_pair = blocks * N2 * sizeof(double2);
  // what the per-time-slice products and co-factors leave of the budget
  const size_t fixed = ((size_t)4 + (g ? 3 : 0)) * Nt * blk16 * sizeof(double2);
  const size_t budget = CHAIN_BUDGET - std::min(CHAIN_BUDGET, fixed);
  const size_t table = 64 * sizeof(DiagTask) + 72 * sizeof(PairTerm) + 5 * sizeof(PairGroup);
  const int batch = (int)std::max<size_t>(1, std::min({pairs.size(), budget / per_pair, TABLE_BUDGET / table}));
  for (const PairBatch& pb : pair_batches(prop, blk16, Nt, 0, Nt, batch, &pairs)) {
    const int np = (int)pb.ent.size();
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get((size_t)np * per_pair, &mem));
    Arena ar;
    ar.base = (double2*)mem;
    ar.N2 = N2;
    auto each = [&](size_t n) {
      std::vector<double2*> v(np);
      for (int i = 0; i < np; i++) v[i] = ar.take(n);
      return v;
    };
    std::vector<double2*> bW, bV;
    for (const auto& m : pb.by_tf) bW.push_back(ar.take(16 * m.size()));
    for (const auto& m : pb.by_ti) bV.push_back(ar.take(32 * m.size()));
    auto Wb = [&](int i, int b, int a) {
      const int h = pb.gtf[i];
      return bW[h] + ((size_t)a * 4 * pb.by_tf[h].size() + pb.ptf[i] * 4 + b) * N2;
    };
    auto Vb = [&](int y, int i, int b) {
      const int h = pb.gti[i];
      return bV[h] + ((size_t)y * 16 * pb.by_ti[h].size() + pb.pti[i] * 16 + b) * N2;
    };
    const std::vector<double2*> bJ = each(16), bP = each(hor ? 32 : 8), bX = each(hor ? 32 : 0),
                                bR = each(g ? 16 : 0), bS = each(g ? 16 : 0), bK = each(g ? 16 : 0),
                                bU = each(g ? 32 : 0), bO = each(g ? 8 : 0), bY = each(g && hor ? 32 : 0),
                                bZ = each(g && hor ? 32 : 0), bQ = each(g && hor ? 32 : 0),
                                bN = each(g && hor ? 8 : 0);
    // blocks (row, column) of the stacked outputs: right block (column) major
    auto rc = [&](double2* b, int r, int col) { return b + (size_t)(col * 4 + r) * N2; };
    // Pm(y): hor: block (a, c) at [c][y * 4 + a]; else the diagonal blocks a at [a][y]
    auto Pm = [&](int y, int i, int a, int c2) {
      return hor ? bP[i] + (size_t)(c2 * 8 + y * 4 + a) * N2 : bP[i] + (size_t)(a * 2 + y) * N2;
    };
    std::vector<GridTask> g0, g1, g2, g3, g4, g5;
    CombList comb;
    for (size_t h = 0; h < pb.by_tf.size(); h++) {
      const std::vector<int>& mi = pb.by_tf[h];
      const int m = (int)mi.size(), tf = pb.tf[mi[0]];
      // W = T^dag L: slab (pair, row b), right block a
      GridTask G = make_grid(4 * m, 4, 4, kOne, 0xF, 0);
      for (int pp = 0; pp < m; pp++)
        for (int b = 0; b < 4; b++)
          for (int k = 0; k < 4; k++) G.A[(size_t)(pp * 4 + b) * 4 + k] = pb.T[mi[pp]] + (size_t)(k * 4 + b) * N2;
      for (int j = 0; j < 4; j++) {
        for (int k = 0; k < 4; k++) G.B[j][k] = M[(size_t)cL * Nt + tf] + (size_t)(k * 4 + j) * N2;
        G.C0[j] = bW[h] + (size_t)j * 4 * m * N2;
      }
      g0.push_back(std::move(G));
    }
    for (size_t h = 0; h < pb.by_ti.size(); h++) {
      const std::vector<int>& mi = pb.by_ti[h];
      const int m = (int)mi.size(), ti = pb.ti[mi[0]];
      // V(y) = tau_b P_y(ti): slab (pair, block b), right block y
      GridTask G = make_grid(16 * m, 2, 1, kOne, 0, 0);
      for (int pp = 0; pp < m; pp++)
        for (int b = 0; b < 16; b++) G.A[pp * 16 + b] = pb.T[mi[pp]] + (size_t)b * N2;
      for (int y = 0; y < 2; y++) {
        G.B[y][0] = P(P1 + y, ti);
        G.C0[y] = bV[h] + (size_t)y * 16 * m * N2;
      }
      g0.push_back(std::move(G));
    }
    for (int i = 0; i < np; i++) {
      const int tf = pb.tf[i], ti = pb.ti[i];
      const double2* T = pb.T[i];
      const double2* wp = w + (size_t)pairs[pb.ent[i]] * 5;
      {  // J = W G T (the trailing G is a sign of its column): slab b, right block d
        GridTask G = make_grid(4, 4, 4, kG5, 0, 0);
        for (int b = 0; b < 4; b++)
          for (int k = 0; k < 4; k++) G.A[b * 4 + k] = Wb(i, b, k);
        for (int j = 0; j < 4; j++) {
          for (int k = 0; k < 4; k++) G.B[j][k] = T + (size_t)(k * 4 + j) * N2;
          G.C0[j] = rc(bJ[i], 0, j);
        }
        g1.push_back(std::move(G));
      }
      if (hor) {  // Pm(y) = V(y) T^dag: slab (y, a), right block c
        GridTask G = make_grid(8, 4, 4, kOne, 0, 0xFFFF);
        for (int y = 0; y < 2; y++)
          for (int a = 0; a < 4; a++)
            for (int k = 0; k < 4; k++) G.A[(size_t)(y * 4 + a) * 4 + k] = Vb(y, i, a * 4 + k);
        for (int j = 0; j < 4; j++) {
          for (int k = 0; k < 4; k++) G.B[j][k] = T + (size_t)(j * 4 + k) * N2;
          G.C0[j] = bP[i] + (size_t)j * 8 * N2;
        }
        g1.push_back(std::move(G));
        for (int y = 0; y < 2; y++) {
          // X(1) = P3 Pm(1), X(2) = P4 Pm(2): block (a, c) at [a * 4 + c]
          for (int jb = 0; jb < 2; jb++) {
            GridTask H = make_grid(1, 8, 1, kOne, 0, 0);
            H.A[0] = P(P3 + y, tf);
            for (int j = 0; j < 8; j++) {
              const int b = 8 * jb + j;
              H.B[j][0] = Pm(y, i, b / 4, b % 4);
              H.C0[j] = bX[i] + (size_t)(y * 16 + b) * N2;
            }
            g2.push_back(std::move(H));
          }
          if (!g) continue;
          // Y(1) = Pm(1) P4, Y(2) = Pm(2) P3; Z(1) = X(2) P3, Z(2) = X(1) P4
          GridTask Y = make_grid(16, 1, 1, kOne, 0, 0), Z = make_grid(16, 1, 1, kOne, 0, 0);
          for (int b = 0; b < 16; b++) {
            Y.A[b] = Pm(y, i, b / 4, b % 4);
            Z.A[b] = bX[i] + (size_t)((1 - y) * 16 + b) * N2;
          }
          Y.B[0][0] = P(y ? P3 : P4, tf);
          Z.B[0][0] = P(y ? P4 : P3, tf);
          Y.C0[0] = bY[i] + (size_t)y * 16 * N2;
          Z.C0[0] = bZ[i] + (size_t)y * 16 * N2;
          g2.push_back(std::move(Y));
          g3.push_back(std::move(Z));
        }
        if (g) {
          // Q(h)_{b u} = sum_v tau_vb^dag Z(h)_{v u}: slab b, right block (h, u)
          GridTask Q = make_grid(4, 8, 4, kOne, 0xF, 0);
          for (int b = 0; b < 4; b++)
            for (int v = 0; v < 4; v++) Q.A[b * 4 + v] = T + (size_t)(v * 4 + b) * N2;
          for (int j = 0; j < 8; j++) {
            for (int v = 0; v < 4; v++) Q.B[j][v] = bZ[i] + (size_t)((j / 4) * 16 + v * 4 + j % 4) * N2;
            Q.C0[j] = bQ[i] + (size_t)j * 4 * N2;
          }
          g4.push_back(std::move(Q));
          // N(h) = sum_u N(h)_u, N(h)_u = sum_b Q(h)_{b u} tau_ub: slab h
          for (int u = 0; u < 4; u++) {
            GridTask G = make_grid(2, 1, 4, kOne, 0, 0);
            for (int h = 0; h < 2; h++)
              for (int b = 0; b < 4; b++) G.A[h * 4 + b] = bQ[i] + (size_t)((h * 4 + u) * 4 + b) * N2;
            for (int b = 0; b < 4; b++) G.B[0][b] = T + (size_t)(u * 4 + b) * N2;
            G.C0[0] = bN[i] + (size_t)u * 2 * N2;
            g5.push_back(std::move(G));
          }
        }
      } else {  // the diagonal blocks Pm(y)_aa alone: slab y
        for (int a = 0; a < 4; a++) {
          GridTask G = make_grid(2, 1, 4, kOne, 0, 0xF);
          for (int y = 0; y < 2; y++)
            for (int k = 0; k < 4; k++) G.A[y * 4 + k] = Vb(y, i, a * 4 + k);
          for (int k = 0; k < 4; k++) G.B[0][k] = T + (size_t)(a * 4 + k) * N2;
          G.C0[0] = Pm(0, i, a, a);
          g1.push_back(std::move(G));
        }
      }
      if (!g) continue;
      // Rw = w_sq Rsq + w_dt Rdt, S = T G Rw, K = S T^dag (the leading G is a sign of its row)
      const double2 a = make_double2(wp[0].x * wdown * wsq, wp[0].y * wdown * wsq),
                    b = make_double2(wp[1].x * wdown * wdt, wp[1].y * wdown * wdt);
      for (int k = 0; k < 16; k++) {
        comb.begin(bR[i] + (size_t)k * N2, false);
        comb.term(M[(size_t)cSq * Nt + ti] + (size_t)k * N2, a);
        comb.term(M[(size_t)cDt * Nt + ti] + (size_t)k * N2, b);
      }
      GridTask S = make_grid(4, 4, 4, kG5, 0, 0), K = make_grid(4, 4, 4, kOne, 0, 0xFFFF);
      for (int r = 0; r < 4; r++)
        for (int k = 0; k < 4; k++) {
          S.A[r * 4 + k] = T + (size_t)(r * 4 + k) * N2;
          K.A[r * 4 + k] = rc(bS[i], r, k);
        }
      for (int j = 0; j < 4; j++) {
        for (int k = 0; k < 4; k++) {
          S.B[j][k] = bR[i] + (size_t)(k * 4 + j) * N2;
          K.B[j][k] = T + (size_t)(j * 4 + k) * N2;
        }
        S.C0[j] = rc(bS[i], 0, j);
        K.C0[j] = rc(bK[i], 0, j);
      }
      g0.push_back(std::move(S));
      g1.push_back(std::move(K));
      // U(x) = P_x tau_b (x = P3, P4): slab x, right block b; O(x)_a = sum_b tau_ab^dag U(x)_ab: right block x
      for (int jb = 0; jb < 2; jb++) {
        GridTask U = make_grid(2, 8, 1, kOne, 0, 0);
        U.A[0] = P(P3, tf);
        U.A[1] = P(P4, tf);
        for (int j = 0; j < 8; j++) {
          U.B[j][0] = T + (size_t)(8 * jb + j) * N2;
          U.C0[j] = bU[i] + (size_t)(8 * jb + j) * 2 * N2;
        }
        g0.push_back(std::move(U));
      }
      for (int r = 0; r < 4; r++) {
        GridTask O = make_grid(1, 2, 4, kOne, 0xF, 0);
        for (int k = 0; k < 4; k++) O.A[k] = T + (size_t)(r * 4 + k) * N2;
        for (int x = 0; x < 2; x++) {
          for (int k = 0; k < 4; k++) O.B[x][k] = bU[i] + (size_t)((r * 4 + k) * 2 + x) * N2;
          O.C0[x] = bO[i] + (size_t)(x * 4 + r) * N2;
        }
        g1.push_back(std::move(O));
      }
    }
    CTR_TRY(comb.run((int)N2, c.s));
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(run_grids(c, g1, WS_TASKS));
    CTR_TRY(run_grids(c, g2, WS_TASKS));
    CTR_TRY(run_grids(c, g3, WS_TASKS));
    CTR_TRY(run_grids(c, g4, WS_TASKS));
    CTR_TRY(run_grids(c, g5, WS_TASKS));
    // ---- values: 64 traces a pair, then the correlators and the twins' weights
    static const int tx[4] = {P4, P3, P3, P4}, ty[4] = {0, 1, 0, 1};  // twins (P4, P1), (P3, P2), (P3, P1), (P4, P2)
    void *dv, *dw[2];
    CTR_TRY(workspace(WS_ROWABS).get((size_t)np * 68 * sizeof(double2), &dv));
    double2* vals = (double2*)dv;
    double2* wk = vals + (size_t)np * 64;
    if (!hor) CTR_CUDA(cudaMemsetAsync(vals, 0, (size_t)np * 64 * sizeof(double2), c.s));
    std::vector<DiagTask> vt;
    PairList pl;
    auto value = [&](const double2* x, const double2* y, int slot) {
      DiagTask d;
      std::memset(&d, 0, sizeof(d));
      d.x = x;
      d.y = y;
      d.out = -1;
      d.vout = slot;
      vt.push_back(d);
    };
    std::vector<int> ent(np);
    std::vector<double2> wsf((size_t)np * 2);
    for (int i = 0; i < np; i++) {
      const int v0 = i * 64, ti = pb.ti[i], tf = pb.tf[i];
      ent[i] = pairs[pb.ent[i]];
      const double2* wp = w + (size_t)ent[i] * 5;
      wsf[2 * i] = make_double2(wp[2].x * wst, wp[2].y * wst);
      wsf[2 * i + 1] = make_double2(wp[3].x * wfi, wp[3].y * wfi);
      for (int b = 0; b < 16; b++) {
        // Tr[R_{a b} J_{b a}] g5(a)
        value(M[(size_t)cSq * Nt + ti] + (size_t)b * N2, rc(bJ[i], b % 4, b / 4), v0 + b);
        value(M[(size_t)cDt * Nt + ti] + (size_t)b * N2, rc(bJ[i], b % 4, b / 4), v0 + 16 + b);
        if (hor)
          value(bX[i] + (size_t)b * N2, bX[i] + (size_t)(16 + (b % 4) * 4 + b / 4) * N2, v0 + 32 + b);
      }
      for (int k = 0; k < 4; k++)
        for (int a = 0; a < 4; a++) value(P(tx[k], tf), Pm(ty[k], i, a, a), v0 + 48 + k * 4 + a);
      if (!g) continue;
      if (hor) {
        pl.begin(make_double2(wp[4].x * wdh, wp[4].y * wdh));
        for (int b = 0; b < 16; b++) {
          const int bt = (b % 4) * 4 + b / 4;
          pl.term(bX[i] + (size_t)b * N2, bX[i] + (size_t)(16 + bt) * N2);
          pl.term(bY[i] + (size_t)b * N2, bY[i] + (size_t)(16 + bt) * N2);
        }
        for (int y = 0; y < 2; y++)
          for (int u = 0; u < 4; u++) pl.term(P(P1 + y, ti), bN[i] + (size_t)(u * 2 + y) * N2);
      }
      for (int k = 0; k < 4; k++) {
        pl.begin(make_double2(1.0, 0.0), wk + 4 * (size_t)i + k);
        for (int a = 0; a < 4; a++) {
          pl.term(P(tx[k], tf), Pm(ty[k], i, a, a));
          pl.term(P(P1 + ty[k], ti), bO[i] + (size_t)((tx[k] - P3) * 4 + a) * N2);
        }
      }
    }
    CTR_TRY(launch_diag(vt, 0, N, f, vals, nullptr, c.s));
    CTR_TRY(upload_group(WS_MISC, {{ent.data(), ent.size() * sizeof(int)}, {wsf.data(), wsf.size() * sizeof(double2)}},
                         dw, c.s));
    {
      TimedLaunch tl(c.s, "pipi_combine");
      pipi_vjp_combine_kernel<<<(np + 127) / 128, 128, 0, c.s>>>(vals, (const int*)dw[0], (const double2*)dw[1], np, wsq,
                                                                 wdt, wst, wfi, wdh, corr, wk);
      CTR_CUDA(cudaGetLastError());
    }
    CTR_TRY(pl.run(N, f, nullptr, grad, c.s));
    if (!g) continue;
    // ---- co-factors of the batch, summed per time slice
    CombList sum;
    for (const std::vector<int>& mi : pb.by_tf)
      for (int b = 0; b < 16; b++) {
        sum.begin(Ks + (size_t)pb.tf[mi[0]] * blk16 + (size_t)b * N2, true);
        for (int i : mi) sum.term(rc(bK[i], b / 4, b % 4), make_double2(1.0, 0.0));
      }
    for (const std::vector<int>& mi : pb.by_ti)
      for (int k = 0; k < 2; k++)
        for (int b = 0; b < 16; b++) {
          sum.begin((k ? Jd : Js) + (size_t)pb.ti[mi[0]] * blk16 + (size_t)b * N2, true);
          for (int i : mi) {
            const double2 wv = w[(size_t)pairs[pb.ent[i]] * 5 + k];
            const double sc = k ? wdt : wsq;
            sum.term(rc(bJ[i], b / 4, b % 4), make_double2(wv.x * wdown * sc, wv.y * wdown * sc));
          }
        }
    CTR_TRY(sum.run((int)N2, c.s));
  }
  if (!g) return CTR_OK;
  // ---- per time slice: Tr[Pa tau_ab Pb F_ba] with co-factor F = K (L at the sink times) and Jsq, Jdt (R at the
  // source times): (tau Pb)(F Pa) holds the right indices, (Pa tau)(Pb F) the left ones
  struct Slice {
    int t, a, b;
    const double2* F;
    bool row_sign;  // gamma_5 on F's row (K) or its column (J)
  };
  std::vector<Slice> sl;
  for (int t = 0; t < Nt; t++) {
    if (on_tf[t]) sl.push_back({t, P3, P4, Ks + (size_t)t * blk16, true});
    if (on_ti[t]) {
      sl.push_back({t, P2, P1, Js + (size_t)t * blk16, false});
      sl.push_back({t, P1, P2, Jd + (size_t)t * blk16, false});
    }
  }
  const size_t per_sl = 64 * N2 * sizeof(double2);
  const size_t chunk = std::max<size_t>(1, std::min(sl.size(), budget / per_sl));
  for (size_t s0 = 0; s0 < sl.size(); s0 += chunk) {
    const size_t ns = std::min(chunk, sl.size() - s0);
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get(ns * per_sl, &mem));
    std::vector<GridTask> g0;
    PairList pl;
    for (size_t k = 0; k < ns; k++) {
      const Slice& S = sl[s0 + k];
      const double2* D = prop + (size_t)S.t * (Nt + 1) * blk16;
      double2* o = (double2*)mem + k * 64 * N2;  // tau Pb, F Pa, Pa tau, Pb F
      GridTask A = make_grid(16, 1, 1, kOne, 0, 0), B = make_grid(16, 1, 1, kOne, 0, 0);
      for (int b = 0; b < 16; b++) {
        A.A[b] = D + (size_t)b * N2;
        B.A[b] = S.F + (size_t)b * N2;
      }
      A.B[0][0] = P(S.b, S.t);
      B.B[0][0] = P(S.a, S.t);
      A.C0[0] = o;
      B.C0[0] = o + blk16;
      g0.push_back(std::move(A));
      g0.push_back(std::move(B));
      for (int jb = 0; jb < 2; jb++) {
        GridTask C = make_grid(1, 8, 1, kOne, 0, 0), E = make_grid(1, 8, 1, kOne, 0, 0);
        C.A[0] = P(S.a, S.t);
        E.A[0] = P(S.b, S.t);
        for (int j = 0; j < 8; j++) {
          C.B[j][0] = D + (size_t)(8 * jb + j) * N2;
          E.B[j][0] = S.F + (size_t)(8 * jb + j) * N2;
          C.C0[j] = o + 2 * blk16 + (size_t)(8 * jb + j) * N2;
          E.C0[j] = o + 3 * blk16 + (size_t)(8 * jb + j) * N2;
        }
        g0.push_back(std::move(C));
        g0.push_back(std::move(E));
      }
      pl.begin(make_double2(1.0, 0.0), nullptr, wup);
      for (int b = 0; b < 16; b++) {
        const int bt = (b % 4) * 4 + b / 4;  // tau_ab against F_ba
        const int u = G5[S.row_sign ? b % 4 : b / 4] < 0 ? 2 : 0;
        pl.term(o + (size_t)b * N2, o + blk16 + (size_t)bt * N2, u);
        pl.term(o + 2 * blk16 + (size_t)b * N2, o + 3 * blk16 + (size_t)bt * N2, u);
      }
    }
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(pl.run(N, f, nullptr, grad, c.s));
  }
  return CTR_OK;
}

}  // namespace

int chain_values(int N, int Nt, int nphi, const double* prop, const double* phi, const std::vector<ctr_factor>& factors,
                 const std::vector<int>& off, double* values, cudaStream_t s, int engine) {
  ChainRunner R(N, Nt, nphi, (const double2*)prop, (const double2*)phi, nullptr, (double2*)values, nullptr, s, engine);
  const int nchain = (int)off.size() - 1;
  for (int c = 0; c < nchain; c++) {
    const int n = off[c + 1] - off[c];
    if (n < 2 || n > CTR_CHAIN_MAXF) return fail(CTR_ERR_ARG, "chain %d has %d factors", c, n);
    for (int j = 0; j < n; j++) CTR_TRY(R.check(factors[off[c] + j]));
    CTR_TRY(R.add(&factors[off[c]], n, make_double2(0.0, 0.0), c, false));
    CTR_TRY(R.end_group());
  }
  return R.flush();
}

}  // namespace ctr

using namespace ctr;

extern "C" {

int ctr_apply_profile(int nev, long long nmat, const double* f, const double* src, double* dst, void* stream) {
  if (nev < 1 || nmat < 0 || !f || !src || !dst) return fail(CTR_ERR_ARG, "ctr_apply_profile: bad arguments");
  if (nmat == 0) return CTR_OK;
  TimedLaunch tl((cudaStream_t)stream, "apply_profile");
  apply_profile_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>((const double2*)src, (double2*)dst, f, nev, nmat);
  CTR_CUDA(cudaGetLastError());
  return CTR_OK;
}

int ctr_chain_adjoint(int engine, int nev, int nt, int nphi, const double* prop, const double* phi, const double* f,
                      int nchain, const int* chain_off, const ctr_factor* factors, const double* w, double* values,
                      double* grad, void* stream) {
  CTR_NO_CAPTURE("ctr_chain_adjoint");
  cudaStream_t s = (cudaStream_t)stream;
  CTR_TRY(check_engine(engine, nev));
  if (nev < 1 || nt < 1 || nphi < 0 || nchain < 0 || !prop || !f || !chain_off || !factors || (!values && !grad))
    return fail(CTR_ERR_ARG, "ctr_chain_adjoint: bad arguments");
  if (grad && !w) return fail(CTR_ERR_ARG, "ctr_chain_adjoint: weights are needed for the gradient");
  if (nphi > 0 && !phi) return fail(CTR_ERR_ARG, "ctr_chain_adjoint: elementals missing");
  CTR_TRY(check_f(nev, f, s));
  double2* phis = nullptr;
  if (nphi > 0) CTR_TRY(profiled(nev, (long long)nt * nphi, phi, f, WS_PHI, &phis, s));
  ChainRunner R(nev, nt, nphi, (const double2*)prop, phis, f, (double2*)values, grad, s, engine);
  for (int c = 0; c < nchain; c++) {
    const int n = chain_off[c + 1] - chain_off[c];
    if (n < 2 || n > CTR_CHAIN_MAXF) return fail(CTR_ERR_ARG, "chain %d has %d factors (2..%d)", c, n, CTR_CHAIN_MAXF);
    for (int j = 0; j < n; j++) CTR_TRY(R.check(factors[chain_off[c] + j]));
    const double2 wc = w ? make_double2(w[2 * c], w[2 * c + 1]) : make_double2(0.0, 0.0);
    CTR_TRY(R.add(factors + chain_off[c], n, wc, values ? c : -1, grad != nullptr));
    CTR_TRY(R.end_group());
  }
  return R.flush();
}

int ctr_rho_profile_vjp(int engine, int nev, int nt, const double* prop, const double* mom5, const double* f,
                        const double* w, double* corr, double* grad, void* stream) {
  CTR_NO_CAPTURE("ctr_rho_profile_vjp");
  cudaStream_t s = (cudaStream_t)stream;
  CTR_TRY(check_engine(engine, nev));
  if (nev < 1 || nt < 1 || !prop || !mom5 || !f || !w || (!corr && !grad))
    return fail(CTR_ERR_ARG, "ctr_rho_profile_vjp: bad arguments");
  CTR_TRY(check_f(nev, f, s));
  std::vector<double> hw((size_t)nt * nt * 48 * 2);
  CTR_CUDA(cudaMemcpyAsync(hw.data(), w, hw.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  CTR_CUDA(cudaStreamSynchronize(s));
  double2* phis;
  CTR_TRY(profiled(nev, (long long)nt * 5, mom5, f, WS_PHI, &phis, s));
  CorrOut out(corr, (size_t)nt * nt * 48);
  CTR_TRY(out.open());
  CTR_TRY(rho_vjp(Ctx{nev, nt, (size_t)nev * nev, s, engine, true}, (const double2*)prop, phis, f, (const double2*)hw.data(),
                  out.p, grad));
  return out.close(s);
}

int ctr_pipi_profile_vjp(int engine, int nev, int nt, int isospin, const double* prop, const double* p1,
                         const double* p2, const double* p3, const double* p4, const double* f, const double* w,
                         double* corr, double* grad, void* stream) {
  CTR_NO_CAPTURE("ctr_pipi_profile_vjp");
  cudaStream_t s = (cudaStream_t)stream;
  CTR_TRY(check_engine(engine, nev));
  if (nev < 1 || nt < 1 || !prop || !p1 || !p2 || !p3 || !p4 || !f || !w || (!corr && !grad))
    return fail(CTR_ERR_ARG, "ctr_pipi_profile_vjp: bad arguments");
  if (isospin != 0 && isospin != 1) return fail(CTR_ERR_ARG, "isospin must be 0 (I=0) or 1 (I=1)");
  CTR_TRY(check_f(nev, f, s));
  std::vector<double> hw((size_t)nt * nt * 5 * 2);
  CTR_CUDA(cudaMemcpyAsync(hw.data(), w, hw.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  CTR_CUDA(cudaStreamSynchronize(s));
  // the distinct elementals, profiled: [elemental][t]
  int32_t set[4];
  std::vector<Elem> el = elems(nev, {p1, p2, p3, p4}, set);
  const size_t n1 = (size_t)nt * nev * nev;
  void* mem;
  CTR_TRY(workspace(WS_PHI).get(el.size() * n1 * sizeof(double2), &mem));
  for (size_t k = 0; k < el.size(); k++) {
    if (!aligned16(el[k].p)) {  // p1..p4 need only hold doubles
      void* raw;
      CTR_TRY(workspace(WS_SCRATCH).get(n1 * sizeof(double2), &raw));
      CTR_CUDA(cudaMemcpyAsync(raw, el[k].p, n1 * sizeof(double2), cudaMemcpyDeviceToDevice, s));
      el[k].p = (const double2*)raw;
    }
    TimedLaunch tl(s, "apply_profile");
    apply_profile_kernel<<<1024, 256, 0, s>>>(el[k].p, (double2*)mem + k * n1, f, nev, nt);
    CTR_CUDA(cudaGetLastError());
    el[k].p = (const double2*)mem + k * n1;
  }
  CorrOut out(corr, (size_t)nt * nt * 5);
  CTR_TRY(out.open());
  CTR_TRY(pipi_vjp(Ctx{nev, nt, (size_t)nev * nev, s, engine, true}, isospin, (const double2*)prop, el, set, f,
                   (const double2*)hw.data(), out.p, grad));
  return out.close(s);
}

}  // extern "C"
