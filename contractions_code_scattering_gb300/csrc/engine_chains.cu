// Chain diagrams: rho->pipi, pipi->pipi (I=1, I=0), loop-unity, sigma->pipi,
// on either engine: every GEMM stage below is a list of block products that runs on
// the FP64 tile kernel or on the split-precision tensor-core engine.  The closing
// traces are FP64 on both, but for the momentum-set calls of rho->pipi and sigma->pipi
// on the split engine, which take them as Gram products.
//
// The reference evaluates every spin row as an independent chain of 2-6 Nev^3
// products (lib/calculate_{rhopi,pipi_*,sigmapi_*,loop_unity}_core.h).  The
// tables are gamma_5-diagonal in the summed indices, so the spin sums factor
// into 4x4 spin-block matrix products, with G = diag(gamma_5) x 1:
//   R(t)  = Phi_a(t) tau(t,t)_{..} Phi_b(t)                     (per time slice)
//   L(t)  = Phi3(t) tau(t,t)_{..} Phi4(t)
//   square(tf,ti) = Tr[G S W],  S = T G Rsq,  W = T^dag L,  Rsq = Phi2 taud Phi1
//   dtri(tf,ti)   = Tr[G S W],  S = T G Rdt,                Rdt = Phi1 taud Phi2
//   dtri_hor      = Tr[Phi3 Pm(1) Phi4 Pm(2)],  Pm(q) = T Phi_q T^dag
//   star / fish   = products of twin traces sum_b Tr[(tau_b Phi_y(ti)) (tau_b^dag Phi_x(tf))]
//   rho->pipi     = sum c * Tr[Phi_ip (T G R)_{s5 s2} tau_{s3 s2}^dag]
//   sigma->pipi triangle = sum g5(s1) Tr[Phi_ik (T G R)_{s1 s5} tau_{s1 s5}^dag]
// with T = tau(tf,ti) as a 4x4 block matrix.  S depends on the source side only
// and W on the sink side only, so momentum sets share them: the square of the
// set (p, -p) and the double triangle of (-p, p) have one S.  Each block product
// is one task of the batched GEMM (up to 4 accumulated terms with the gamma_5
// signs).
#include <algorithm>
#include <array>
#include <cstring>
#include <iterator>
#include <map>
#include <tuple>
#include <utility>

#include "chains.h"

namespace ctr {

// Stage = one launch of the batched GEMM; stages run in order on the stream.
int run_stage(const Ctx& c, const std::vector<ZTask>& tasks, int slot) {
  if (tasks.empty()) return CTR_OK;
  if (c.engine == CTR_ENGINE_SPLIT) return zgemm_split_tasks(c.N, tasks.data(), (int)tasks.size(), c.s);
  void* d;
  CTR_TRY(upload(slot, tasks.data(), tasks.size() * sizeof(ZTask), &d, c.s));
  return launch_zgemm_f64((const ZTask*)d, (int)tasks.size(), c.N, c.s, tasks.data());
}

int run_traces(const Ctx& c, const std::vector<TraceTask>& t) {
  if (t.empty()) return CTR_OK;
  void* d;
  CTR_TRY(upload(WS_ROWTASKS, t.data(), t.size() * sizeof(TraceTask), &d, c.s));
  return launch_trace_f64((const TraceTask*)d, (int)t.size(), c.N, c.s);
}

// A stage of block grids: the split engine stacks each grid's slabs along M; the
// FP64 engine runs them as plain tasks.
int run_grids(const Ctx& c, const std::vector<GridTask>& g, int slot) {
  if (g.empty()) return CTR_OK;
  if (c.engine == CTR_ENGINE_SPLIT) return zgemm_split_grids(c.N, g, c.s, c.full);
  std::vector<ZTask> t;
  for (const GridTask& G : g)
    for (int sl = 0; sl < G.nslab; sl++)
      for (int j = 0; j < G.nb; j++) {
        ZTask z{};
        for (int q = 0; q < G.nterm; q++) {
          z.A[q] = G.A[(size_t)sl * G.nterm + q];
          z.B[q] = G.B[j][q];
          z.wre[q] = G.w[q];
        }
        z.nterm = G.nterm;
        z.flags = G.adag | (((G.bdag >> (4 * j)) & 0xF) << 4);
        z.C = G.C0[j] + (size_t)sl * c.N2;
        t.push_back(z);
      }
  return run_stage(c, t, slot);
}

static inline TraceTask tr(const double2* X, const double2* Y, double2* out, float cre, float cim, int mode) {
  TraceTask t{};
  t.X = X;
  t.Y = Y;
  t.out = out;
  t.coef[0] = cre;
  t.coef[1] = cim;
  t.mode = mode;
  return t;
}

GridTask make_grid(int nslab, int nb, int nterm, const float* w, int adag, int bdag) {
  GridTask G;
  std::memset(G.B, 0, sizeof(G.B));
  std::memset(G.C0, 0, sizeof(G.C0));
  for (int q = 0; q < 4; q++) G.w[q] = q < nterm ? w[q] : 0.f;
  G.nslab = nslab;
  G.nb = nb;
  G.nterm = nterm;
  G.adag = adag;
  G.bdag = bdag;
  G.A.resize((size_t)nslab * nterm);
  return G;
}

std::vector<PairBatch> pair_batches(const double2* tau, size_t blk16, int Nt, int tf_begin, int rows, int batch,
                                    const std::vector<int>* plist, int hmax) {
  std::vector<std::vector<std::pair<int, int>>> out;  // (position, pair)
  if (plist) {
    for (size_t i = 0; i < plist->size(); i++) {
      if (i % batch == 0) out.emplace_back();
      out.back().push_back({(int)i, (*plist)[i]});
    }
  } else {
    int h = rows;
    if ((long long)rows * Nt > batch) {
      int e = 1;
      while ((e + 1) * (e + 1) <= batch) e++;
      h = std::min(rows, e >= 16 ? e & ~7 : e);
    }
    h = std::min(h, hmax);
    const int w = std::min(Nt, std::max(1, batch / h));
    for (int f0 = 0; f0 < rows; f0 += h)
      for (int t0 = 0; t0 < Nt; t0 += w) {
        out.emplace_back();
        for (int ti = t0; ti < std::min(Nt, t0 + w); ti++)
          for (int tfl = f0; tfl < std::min(rows, f0 + h); tfl++)
            out.back().push_back({tfl * Nt + ti, tfl * Nt + ti});
      }
  }
  std::vector<PairBatch> res;
  for (auto& o : out) {
    PairBatch b;
    std::map<int, int> mi, mf;
    for (auto& e : o) {
      const int tfl = e.second / Nt, ti = e.second % Nt, i = (int)b.ent.size();
      b.ent.push_back(e.first);
      b.tf.push_back(tf_begin + tfl);
      b.ti.push_back(ti);
      b.T.push_back(tau + ((size_t)tfl * Nt + ti) * blk16);
      auto place = [&](std::map<int, int>& m, std::vector<std::vector<int>>& groups, int t, std::vector<int>& g,
                       std::vector<int>& pos) {
        auto it = m.emplace(t, (int)groups.size()).first;
        if (it->second == (int)groups.size()) groups.emplace_back();
        g.push_back(it->second);
        pos.push_back((int)groups[it->second].size());
        groups[it->second].push_back(i);
      };
      place(mi, b.by_ti, ti, b.gti, b.pti);
      place(mf, b.by_tf, tfl, b.gtf, b.ptf);
    }
    res.push_back(std::move(b));
  }
  return res;
}

namespace {

// ---- per-entry refinement of split-engine chains
// A chain entry's rounding error is estimated as REFINE_EPS_CHAIN times the sum
// of |coef| sum |Y|_1 |T|_1 over its closing traces (for products of traces,
// the product rule of those scales).  The chain products run on the
// high-precision split configuration (6 slices, levels 0-3 exact, exact integer
// recombination), which keeps ~2^-53 of their row/column scales.  Measured on
// the 20 480 entries of one pi pi momentum pair at Nev=100, Lt=64 against the
// FP64 engine, the largest entry error without any refinement was 1.8e-10;
// with REFINE_EPS_CHAIN = 2^-52 no entry is flagged there, and the check stays
// as the safety net for entries whose cancellation exceeds ~10^6.
constexpr double REFINE_EPS_CHAIN = 1.0 / 4503599627370496.0;  // 2^-52

struct Refine {
  bool on = false;
  double eps_over_tol = 0.0;
  int* count = nullptr;
  int* list = nullptr;
};

int refine_begin(const Ctx& c, size_t nentries, int slot, Refine& r) {
  r.on = c.engine == CTR_ENGINE_SPLIT && g_refine_tol > 0.0;
  if (!r.on) return CTR_OK;
  r.eps_over_tol = REFINE_EPS_CHAIN / g_refine_tol;
  void* p;
  CTR_TRY(workspace(slot).get((nentries + 1) * sizeof(int), &p));
  r.count = (int*)p;
  r.list = r.count + 1;
  CTR_CUDA(cudaMemsetAsync(r.count, 0, sizeof(int), c.s));
  return CTR_OK;
}

// Flagged entries e -> units e / nout (pairs or time slices); rerun(units, out,
// stream) writes their FP64 values as [units][nout] into out (device); they are
// then scattered over corr, and their number is added to g_refined_last.  The
// list is read on the host, so under graph recording this runs after the
// recorded kernels at every launch (the closure holds copies of what it needs).
template <typename Rerun>
int refine_end(const Ctx& c, const Refine& r, int nout, int slot, double2* corr, Rerun rerun) {
  if (!r.on) return CTR_OK;
  const int* count = r.count;
  const int* flagged = r.list;
  return host_step(c.s, [=](cudaStream_t s) -> int {
    int n = 0;
    CTR_TRY(download(&n, count, sizeof(int), s));
    if (n == 0) return CTR_OK;
    std::vector<int> list(n);
    CTR_TRY(download(list.data(), flagged, n * sizeof(int), s));
    std::vector<int> units;
    for (int e : list) units.push_back(e / nout);
    std::sort(units.begin(), units.end());
    units.erase(std::unique(units.begin(), units.end()), units.end());
    void* tmp;
    CTR_TRY(workspace(slot).get(units.size() * nout * sizeof(double2), &tmp));
    CTR_TRY(rerun(units, (double2*)tmp, s));
    std::vector<int> where(units.size() * nout);
    for (size_t q = 0; q < units.size(); q++)
      for (int o = 0; o < nout; o++) where[q * nout + o] = units[q] * nout + o;
    void* dw;
    CTR_TRY(upload(WS_TASKS, where.data(), where.size() * sizeof(int), &dw, s));
    CTR_TRY(launch_scatter((const int*)dw, (const double2*)tmp, (int)where.size(), corr, s));
    g_refined_last += (long long)where.size();
    return CTR_OK;
  });
}

// Closing traces of a batch; add() returns the slot of the value.
struct TracePlan {
  std::vector<TraceTask> tt;
  int n = 0;
  bool keep = true;  // false: number the slots only (the traces run in another form)
  int add(const double2* x, const double2* y, float cre, float cim, int mode) {
    if (keep) tt.push_back(tr(x, y, nullptr, cre, cim, mode));
    return n++;
  }
};

// (set, pair) item of a pi pi batch: 112 trace slots (16 each of square, double triangle,
// horizontal double triangle and the four twins; -1: none), combined into corr[ent * 5 ..].
//
// A block of S = T G R or W = T^dag L may cancel in its sum of four terms, and the error
// scales of square and double triangle with it.  They are at least what the sums have
// without cancellation: 0.78^2 / Nev sum_ab (sum_k |T_ak|^2 |R_kb|^2)^(1/2) (sum_c |T_cb|^2
// |L_ca|^2)^(1/2) from the blocks' norms nT (of a pair), nM (of L and R per time slice; row
// terms[4 it] of nT, rows terms[4 it + 1..3] of nM for L, Rsq and Rdt), times the 0.78 that
// a sum of |S| |W| has of the product of their norms.
__global__ void pipi_combine_sets_kernel(const double2* __restrict__ trv, const double* __restrict__ trabs,
                                         const int* __restrict__ slots, const int* __restrict__ ent, int nitem, int iso,
                                         double2* __restrict__ corr, double eps_over_tol, int* __restrict__ count,
                                         int* __restrict__ list, const int* __restrict__ terms,
                                         const double* __restrict__ nT, const double* __restrict__ nM, double per_nev) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= nitem) return;
  const int* sl = slots + (size_t)it * 112;
  double2 sum[7];
  double ab[7];
  for (int g = 0; g < 7; g++) {
    double re = 0, im = 0, a = 0;
    for (int k = 0; k < 16; k++) {
      const int j = sl[g * 16 + k];
      if (j < 0) continue;
      re += trv[j].x;
      im += trv[j].y;
      if (trabs) a += trabs[j];
    }
    sum[g] = make_double2(re, im);
    ab[g] = a;
  }
  if (trabs) {
    const int* m = terms + 4 * (size_t)it;
    const double *T = nT + 16 * (size_t)m[0], *L = nM + 16 * (size_t)m[1];
    for (int g = 0; g < 2; g++) {
      const double* R = nM + 16 * (size_t)m[2 + g];
      double f = 0.0;
      for (int b = 0; b < 16; b++) {
        double es = 0.0, ew = 0.0;
        for (int k = 0; k < 4; k++) {
          const double s = T[(b & 12) + k] * R[4 * k + (b & 3)], w = T[4 * k + (b & 3)] * L[4 * k + (b >> 2)];
          es += s * s;
          ew += w * w;
        }
        f += sqrt(es) * sqrt(ew);
      }
      ab[g] = fmax(ab[g], 0.47 * per_nev * f);
    }
  }
  const double2 star = cmul(sum[3], sum[4]);
  const double2 fish = cmul(sum[5], sum[6]);
  double2* o = corr + (size_t)ent[it] * 5;
  if (iso == 1) {  // lib/contract_kernels_pipi.cu:288-303
    o[0] = make_double2(-2. * sum[0].x, -2. * sum[0].y);
    o[1] = make_double2(2. * sum[1].x, 2. * sum[1].y);
    o[2] = make_double2(-star.x, -star.y);
    o[3] = fish;
    o[4] = make_double2(0., 0.);
  } else {  // lib/contract_kernels_pipi.cu:463-478
    o[0] = make_double2((-1. / 3.) * sum[0].x, (-1. / 3.) * sum[0].y);
    o[1] = make_double2(-(1. / 3.) * sum[1].x, -(1. / 3.) * sum[1].y);
    o[2] = star;
    o[3] = fish;
    o[4] = make_double2(-(5. / 3.) * sum[2].x, -(5. / 3.) * sum[2].y);
  }
  if (trabs && eps_over_tol > 0.0) {
    auto mag = [](double2 v) { return sqrt(v.x * v.x + v.y * v.y); };
    const double w[3] = {iso == 1 ? 2.0 : 1.0 / 3.0, iso == 1 ? 2.0 : 1.0 / 3.0, iso == 1 ? 0.0 : 5.0 / 3.0};
    const double scale[5] = {w[0] * ab[0], w[1] * ab[1], mag(sum[3]) * ab[4] + mag(sum[4]) * ab[3],
                             mag(sum[5]) * ab[6] + mag(sum[6]) * ab[5], w[2] * ab[2]};
    for (int k = 0; k < 5; k++)
      if (!(scale[k] * eps_over_tol <= mag(o[k])) || (scale[k] == 0.0 && mag(o[k]) > 0.0)) {
        list[atomicAdd(count, 1)] = ent[it] * 5 + k;
        break;
      }
  }
}

}  // namespace

// Scratch budget of a set batch: 16 GB, or an eighth of the device's memory where less.
size_t sets_budget() {
  static size_t b = 0;
  if (!b && !capturing()) {
    size_t fr = 0, tot = 0;
    b = cudaMemGetInfo(&fr, &tot) == cudaSuccess ? std::min<size_t>((size_t)16 << 30, tot / 8) : ((size_t)6 << 30);
  }
  return b ? b : ((size_t)6 << 30);
}

// Per time slice: M(a, b, t) = Phi_a(t) taud(t) Phi_b(t), 16 consecutive blocks at
// M[combo * Nt + t], for the (a, b) combos and the t flagged in need.  Two stages
// of grids: Phi_a taud_blk for every a of a time slice stacked along M against
// taud_blk, then its 16 blocks stacked against every Phi_b that follows a.  taud(t) =
// diag + t * dstride.  The time slices run in groups where all their Phi_a taud
// would make it more than `cap` blocks (0: no limit).
int per_t_products(const Ctx& c, const double2* diag, size_t dstride, const std::vector<Elem>& el, int slot,
                   const std::vector<std::pair<int, int>>& combos, const std::vector<std::vector<char>>& need,
                   size_t cap, std::vector<const double2*>& M) {
  const int Nt = c.Nt, nc = (int)combos.size();
  const size_t N2 = c.N2, blk16 = 16 * N2;
  auto P = [&](int q, int t) { return el[q].p + (size_t)t * el[q].stride; };
  M.assign((size_t)nc * Nt, nullptr);
  size_t nblk = 0, ntmp = 0;
  std::vector<std::vector<int>> as(Nt);  // distinct first elementals of each time slice
  for (int t = 0; t < Nt; t++)
    for (int ci = 0; ci < nc; ci++)
      if (need[ci][t]) {
        nblk += 16;
        if (std::find(as[t].begin(), as[t].end(), combos[ci].first) == as[t].end()) as[t].push_back(combos[ci].first);
      }
  const size_t room = cap == 0 ? ~(size_t)0 : cap - std::min(cap, nblk);
  std::vector<int> ends;  // of the groups of time slices
  for (int t = 0, t0 = 0, used = 0; t < Nt; t++) {
    const int n = 16 * (int)as[t].size();
    if (t > t0 && (size_t)(used + n) > room) {
      ends.push_back(t0 = t);
      used = 0;
    }
    used += n;
    ntmp = std::max<size_t>(ntmp, used);
  }
  ends.push_back(Nt);
  void* mem;
  CTR_TRY(workspace(slot).get((nblk + ntmp) * N2 * sizeof(double2), &mem));
  double2 *next = (double2*)mem, *const tmp0 = next + nblk * N2;
  for (size_t e = 0; e < ends.size(); e++) {
    std::vector<GridTask> g0, g1;
    double2* tnext = tmp0;
    for (int t = e ? ends[e - 1] : 0; t < ends[e]; t++) {
      const int na = (int)as[t].size();
      if (!na) continue;
      double2* tmp = tnext;  // block b of the a-th elemental at (b * na + a)
      tnext += (size_t)16 * na * N2;
      for (int jb = 0; jb < 2; jb++) {
        GridTask G = make_grid(na, 8, 1, kOne, 0, 0);
        for (int k = 0; k < na; k++) G.A[k] = P(as[t][k], t);
        for (int j = 0; j < 8; j++) {
          G.B[j][0] = diag + (size_t)t * dstride + (size_t)(8 * jb + j) * N2;
          G.C0[j] = tmp + (size_t)(8 * jb + j) * na * N2;
        }
        g0.push_back(std::move(G));
      }
      for (int k = 0; k < na; k++) {
        std::vector<int> cs;
        for (int ci = 0; ci < nc; ci++)
          if (need[ci][t] && combos[ci].first == as[t][k]) cs.push_back(ci);
        for (size_t c0 = 0; c0 < cs.size(); c0 += 8) {
          GridTask G = make_grid(16, (int)std::min<size_t>(8, cs.size() - c0), 1, kOne, 0, 0);
          for (int b = 0; b < 16; b++) G.A[b] = tmp + ((size_t)b * na + k) * N2;
          for (int j = 0; j < G.nb; j++) {
            const int ci = cs[c0 + j];
            G.B[j][0] = P(combos[ci].second, t);
            G.C0[j] = next;
            M[(size_t)ci * Nt + t] = next;
            next += blk16;
          }
          g1.push_back(std::move(G));
        }
      }
    }
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(run_grids(c, g1, WS_TASKS2));
  }
  return CTR_OK;
}

// Distinct values in ascending order, and the index of each of 0 .. n - 1.
static std::vector<int> index_of(std::vector<int>& v, int n) {
  std::sort(v.begin(), v.end());
  v.erase(std::unique(v.begin(), v.end()), v.end());
  std::vector<int> ix(n, -1);
  for (size_t a = 0; a < v.size(); a++) ix[v[a]] = (int)a;
  return ix;
}

// ------------------------------------------------------------------ pi pi
// Every momentum set (P1..P4 = el[sets[4k ..]]) of one call; with plist, the listed
// pairs only, written in the list's order.  Products that sets share -- R, L, S, W,
// V = tau_b Phi_q, Pm, Phi Pm and the twin traces -- are computed once, whatever
// the number of sets, and a product does not depend on the tile it lands in, so
// each set's entries are bitwise those of a call of its own.
int pipi_core(int N, int Nt, int tf_begin, int tf_end, int iso, const double* prop_rows, const double* prop_diag,
              const std::vector<Elem>& el, int nset, const int32_t* sets, double* corr, cudaStream_t s, int engine,
              bool sets_call, const std::vector<int>* plist) {
  Ctx c{N, Nt, (size_t)N * N, s, engine};
  if (engine == CTR_ENGINE_SPLIT && !plist) g_refined_last = 0;
  const size_t N2 = c.N2, blk16 = 16 * N2;
  const double2 *tau = (const double2*)prop_rows, *diag = (const double2*)prop_diag;
  const int rows = tf_end - tf_begin, npairs = plist ? (int)plist->size() : rows * Nt, nel = (int)el.size();
  auto P = [&](int q, int t) { return el[q].p + (size_t)t * el[q].stride; };
  // ---- per time slice: L = (P3, P4) at the sink times, Rsq = (P2, P1) and Rdt = (P1, P2) at the source times
  std::vector<char> need_tf(Nt, 0), need_ti(Nt, 0);
  for (int i = 0; i < npairs; i++) {
    const int pr = plist ? (*plist)[i] : i;
    need_tf[tf_begin + pr / Nt] = 1;
    need_ti[pr % Nt] = 1;
  }
  Combos cb(Nt);
  std::vector<int> cL(nset), cSq(nset), cDt(nset), CL, CR;
  for (int k = 0; k < nset; k++) {
    const int* q = sets + 4 * k;
    cL[k] = cb.use(q[2], q[3]);
    cSq[k] = cb.use(q[1], q[0]);
    cDt[k] = cb.use(q[0], q[1]);
    for (int t = 0; t < Nt; t++) {
      cb.need[cL[k]][t] |= need_tf[t];
      cb.need[cSq[k]][t] |= need_ti[t];
      cb.need[cDt[k]][t] |= need_ti[t];
    }
    CL.push_back(cL[k]);
    CR.push_back(cSq[k]);
    CR.push_back(cDt[k]);
  }
  std::vector<const double2*> M;
  // a recomputation (plist) keeps its own per-time-slice products
  CTR_TRY(per_t_products(c, diag, blk16, el, plist ? WS_RPHI : WS_PHI, cb.list, cb.need,
                         sets_call ? 0 : 16 * (4 * (size_t)Nt + 4), M));
  const std::vector<int> icl = index_of(CL, (int)cb.list.size()), icr = index_of(CR, (int)cb.list.size());
  const int nCL = (int)CL.size(), nCR = (int)CR.size();
  // elementals on the sink side (P3, P4) and on the source side (P1, P2)
  std::vector<int> Qu, Qw;
  for (int k = 0; k < nset; k++) {
    Qu.push_back(sets[4 * k + 2]);
    Qu.push_back(sets[4 * k + 3]);
    Qw.push_back(sets[4 * k]);
    Qw.push_back(sets[4 * k + 1]);
  }
  const std::vector<int> iu = index_of(Qu, nel), iw = index_of(Qw, nel);
  const int nU = (int)Qu.size(), nW = (int)Qw.size();
  // F = Phi_qf(tf) Pm(qp): per Pm index, the elementals it is multiplied by
  std::vector<std::vector<int>> FK(nW);
  std::vector<int> fpos(nset * 2);
  if (iso == 0)
    for (int k = 0; k < nset; k++)
      for (int h = 0; h < 2; h++) {
        const int qf = sets[4 * k + 2 + h], qp = iw[sets[4 * k + h]];
        auto& v = FK[qp];
        auto it = std::find(v.begin(), v.end(), qf);
        if (it == v.end()) it = v.insert(v.end(), qf);
        fpos[2 * k + h] = (int)(it - v.begin());
      }
  int nF = 0;
  for (auto& v : FK) nF += (int)v.size();
  // star / fish twin traces (sink elemental, source elemental): (4, 1), (3, 2), (3, 1), (4, 2)
  // of every set, a term for each of tau's 16 blocks; on the FP64 engine at I = 0 the 4
  // Tr[Phi_x Pm(y)_cc] instead (Nev = 32, 64 pairs: 6.4 -> 5.9 ms).  The split engine would
  // gain as much (19 sets, Nev = 100, 4 sink times: 165 against 151 ms), but where Pm cancels in
  // its spin sum those traces' error scales fall with it, and entries that need a
  // recomputation go without.
  const bool from_pm = iso == 0 && engine == CTR_ENGINE_FP64;
  std::map<std::pair<int, int>, int> twk;
  std::vector<std::pair<int, int>> TW;
  std::vector<int> twin(4 * nset);
  for (int k = 0; k < nset; k++) {
    const int* q = sets + 4 * k;
    const std::pair<int, int> key[4] = {{q[3], q[0]}, {q[2], q[1]}, {q[2], q[0]}, {q[3], q[1]}};
    for (int h = 0; h < 4; h++) {
      auto it = twk.emplace(key[h], (int)TW.size()).first;
      if (it->second == (int)TW.size()) TW.push_back(key[h]);
      twin[4 * k + h] = it->second;
    }
  }
  const int nTW = (int)TW.size(), ntw = from_pm ? 4 : 16;  // traces a twin
  const size_t blk_pair = 16 * (size_t)(nCR + nCL + nW + (from_pm ? 0 : nU) + (iso == 0 ? nW + nF : 0));
  const size_t tr_pair = (size_t)nset * (iso == 0 ? 48 : 32) + ntw * (size_t)nTW;
  const size_t per_pair = blk_pair * N2 * sizeof(double2) + tr_pair * (sizeof(double2) + sizeof(double));
  const size_t budget = sets_call ? sets_budget() : CHAIN_BUDGET;
  const int batch = std::max(1, std::min(npairs, (int)(budget / std::max<size_t>(per_pair, 1))));
  Refine rf;
  CTR_TRY(refine_begin(c, (size_t)nset * npairs * 5, WS_REFINE, rf));
  double *nM = nullptr, *nT = nullptr;  // norms of L and R (for the call), of T (for a batch)
  if (rf.on) {
    void *p, *d;
    CTR_TRY(workspace(WS_NORMS).get(16 * (M.size() + (size_t)batch) * sizeof(double), &p));
    nM = (double*)p;
    nT = nM + 16 * M.size();
    CTR_TRY(upload(WS_MISC, M.data(), M.size() * sizeof(const double2*), &d, s));
    CTR_TRY(launch_block_norms((const double2* const*)d, (int)M.size(), 16, N, nM, s));
  }
  for (const PairBatch& pb : pair_batches(tau, blk16, Nt, tf_begin, rows, batch, plist)) {
    const int np = (int)pb.ent.size(), ng = (int)pb.by_ti.size(), nh = (int)pb.by_tf.size();
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get((size_t)np * per_pair, &mem));
    double2* base = (double2*)mem;
    size_t used = 0;
    auto alloc = [&](size_t nblk) {
      double2* p = base + used;
      used += nblk * N2;
      return p;
    };
    std::vector<double2*> bS((size_t)ng * nCR), bV(ng), bW((size_t)nh * nCL), bY(nh, nullptr), bP(np, nullptr);
    std::vector<std::vector<double2*>> bF(np, std::vector<double2*>(nW, nullptr));
    for (int g = 0; g < ng; g++) {
      const size_t m = pb.by_ti[g].size();
      for (int ci = 0; ci < nCR; ci++) bS[(size_t)g * nCR + ci] = alloc(16 * m);
      bV[g] = alloc(16 * (size_t)nW * m);
    }
    for (int h = 0; h < nh; h++) {
      const size_t m = pb.by_tf[h].size();
      for (int ci = 0; ci < nCL; ci++) bW[(size_t)h * nCL + ci] = alloc(16 * m);
      if (!from_pm) bY[h] = alloc(16 * (size_t)nU * m);
    }
    for (int i = 0; i < np && iso == 0; i++) {
      bP[i] = alloc(16 * (size_t)nW);
      for (int qp = 0; qp < nW; qp++)
        if (!FK[qp].empty()) bF[i][qp] = alloc(16 * FK[qp].size());
    }
    auto Sblk = [&](int cr, int i, int a, int b) {
      const int g = pb.gti[i];
      return bS[(size_t)g * nCR + icr[cr]] + ((size_t)b * 4 * pb.by_ti[g].size() + pb.pti[i] * 4 + a) * N2;
    };
    auto Wblk = [&](int cl, int i, int b, int a) {
      const int h = pb.gtf[i];
      return bW[(size_t)h * nCL + icl[cl]] + ((size_t)a * 4 * pb.by_tf[h].size() + pb.ptf[i] * 4 + b) * N2;
    };
    auto Vblk = [&](int qi, int i, int b) {
      const int g = pb.gti[i];
      return bV[g] + ((size_t)qi * 16 * pb.by_ti[g].size() + pb.pti[i] * 16 + b) * N2;
    };
    auto Yblk = [&](int qi, int i, int b) {
      const int h = pb.gtf[i];
      return bY[h] + ((size_t)qi * 16 * pb.by_tf[h].size() + pb.ptf[i] * 16 + b) * N2;
    };
    auto Pblk = [&](int qi, int i, int a, int c2) { return bP[i] + ((size_t)c2 * 4 * nW + qi * 4 + a) * N2; };
    std::vector<GridTask> g0, g1, g2;
    for (int g = 0; g < ng; g++) {
      const std::vector<int>& mem_i = pb.by_ti[g];
      const int m = (int)mem_i.size(), ti = pb.ti[mem_i[0]];
      // S = T G R: slab (pair, row block a), right block b of up to two R(t_src) of the call
      for (int c0 = 0; c0 < nCR; c0 += 2) {
        const int nf = std::min(2, nCR - c0);
        GridTask G = make_grid(4 * m, 4 * nf, 4, kG5, 0, 0);
        for (int pp = 0; pp < m; pp++)
          for (int a = 0; a < 4; a++)
            for (int kk = 0; kk < 4; kk++)
              G.A[(size_t)(pp * 4 + a) * 4 + kk] = pb.T[mem_i[pp]] + (size_t)(a * 4 + kk) * N2;
        for (int u = 0; u < nf; u++)
          for (int j = 0; j < 4; j++) {
            for (int kk = 0; kk < 4; kk++)
              G.B[u * 4 + j][kk] = M[(size_t)CR[c0 + u] * Nt + ti] + (size_t)(kk * 4 + j) * N2;
            G.C0[u * 4 + j] = bS[(size_t)g * nCR + c0 + u] + (size_t)j * 4 * m * N2;
          }
        g0.push_back(std::move(G));
      }
      // V(q) = tau_b Phi_q(ti): slab (pair, block b), right block q
      for (int q0 = 0; q0 < nW; q0 += 8) {
        GridTask G = make_grid(16 * m, std::min(8, nW - q0), 1, kOne, 0, 0);
        for (int pp = 0; pp < m; pp++)
          for (int b = 0; b < 16; b++) G.A[pp * 16 + b] = pb.T[mem_i[pp]] + b * N2;
        for (int j = 0; j < G.nb; j++) {
          G.B[j][0] = P(Qw[q0 + j], ti);
          G.C0[j] = bV[g] + (size_t)(q0 + j) * 16 * m * N2;
        }
        g0.push_back(std::move(G));
      }
    }
    for (int h = 0; h < nh; h++) {
      const std::vector<int>& mem_i = pb.by_tf[h];
      const int m = (int)mem_i.size(), tf = pb.tf[mem_i[0]];
      // W = T^dag L: slab (pair, row block b), right block a of up to two L(t_sink) of the call
      for (int c0 = 0; c0 < nCL; c0 += 2) {
        const int nf = std::min(2, nCL - c0);
        GridTask G = make_grid(4 * m, 4 * nf, 4, kOne, 0xF, 0);
        for (int pp = 0; pp < m; pp++)
          for (int b = 0; b < 4; b++)
            for (int kk = 0; kk < 4; kk++)
              G.A[(size_t)(pp * 4 + b) * 4 + kk] = pb.T[mem_i[pp]] + (size_t)(kk * 4 + b) * N2;
        for (int u = 0; u < nf; u++)
          for (int j = 0; j < 4; j++) {
            for (int kk = 0; kk < 4; kk++)
              G.B[u * 4 + j][kk] = M[(size_t)CL[c0 + u] * Nt + tf] + (size_t)(kk * 4 + j) * N2;
            G.C0[u * 4 + j] = bW[(size_t)h * nCL + c0 + u] + (size_t)j * 4 * m * N2;
          }
        g0.push_back(std::move(G));
      }
      // Y(q) = tau_b^dag Phi_q(tf): slab (pair, block b), right block q
      for (int q0 = 0; q0 < nU && !from_pm; q0 += 8) {
        GridTask G = make_grid(16 * m, std::min(8, nU - q0), 1, kOne, 1, 0);
        for (int pp = 0; pp < m; pp++)
          for (int b = 0; b < 16; b++) G.A[pp * 16 + b] = pb.T[mem_i[pp]] + b * N2;
        for (int j = 0; j < G.nb; j++) {
          G.B[j][0] = P(Qu[q0 + j], tf);
          G.C0[j] = bY[h] + (size_t)(q0 + j) * 16 * m * N2;
        }
        g0.push_back(std::move(G));
      }
    }
    for (int i = 0; i < np && iso == 0; i++) {
      // Pm(q) = V(q) T^dag: block (a, c) = sum_k V_ak tau_ck^dag; slab (q, a), right block c
      GridTask gp = make_grid(4 * nW, 4, 4, kOne, 0, 0xFFFF);
      for (int qi = 0; qi < nW; qi++)
        for (int a = 0; a < 4; a++)
          for (int kk = 0; kk < 4; kk++) gp.A[(size_t)(qi * 4 + a) * 4 + kk] = Vblk(qi, i, a * 4 + kk);
      for (int j = 0; j < 4; j++) {
        for (int kk = 0; kk < 4; kk++) gp.B[j][kk] = pb.T[i] + (j * 4 + kk) * N2;
        gp.C0[j] = bP[i] + (size_t)j * 4 * nW * N2;
      }
      g1.push_back(std::move(gp));
      // F(qf, qp)_b = Phi_qf(tf) Pm(qp)_b: slab qf, right block b
      for (int qp = 0; qp < nW; qp++) {
        const int nf = (int)FK[qp].size();
        if (!nf) continue;
        for (int jb = 0; jb < 2; jb++) {
          GridTask gf = make_grid(nf, 8, 1, kOne, 0, 0);
          for (int sl = 0; sl < nf; sl++) gf.A[sl] = P(FK[qp][sl], pb.tf[i]);
          for (int j = 0; j < 8; j++) {
            const int b = 8 * jb + j;
            gf.B[j][0] = Pblk(qp, i, b / 4, b % 4);
            gf.C0[j] = bF[i][qp] + (size_t)b * nf * N2;
          }
          g2.push_back(std::move(gf));
        }
      }
    }
    // the block products run while the host lists the traces
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(run_grids(c, g1, WS_TASKS2));
    CTR_TRY(run_grids(c, g2, WS_GEMM_A));
    // traces: values (and error scales) after the products in the same buffer
    const size_t ntr = (size_t)np * tr_pair;
    double2* trv = base + used;
    double* tra = rf.on ? (double*)(trv + ntr) : nullptr;
    if ((used * sizeof(double2) + ntr * (sizeof(double2) + sizeof(double))) > (size_t)np * per_pair)
      return fail(CTR_ERR_ALLOC, "pi pi: batch arena overflow");
    TracePlan tp;
    tp.tt.reserve(ntr);
    std::vector<int> slots, ent, terms, tws(ntw * (size_t)nTW);
    slots.reserve((size_t)np * nset * 112);
    for (int i = 0; i < np; i++) {
      for (int t = 0; t < nTW; t++)
        for (int b = 0; b < ntw; b++)
          tws[t * ntw + b] = from_pm ? tp.add(P(TW[t].first, pb.tf[i]), Pblk(iw[TW[t].second], i, b, b), 1.f, 0.f, 1)
                                     : tp.add(Vblk(iw[TW[t].second], i, b), Yblk(iu[TW[t].first], i, b), 1.f, 0.f, 1);
      for (int k = 0; k < nset; k++) {
        const int* q = sets + 4 * k;
        for (int cr : {cSq[k], cDt[k]})
          for (int b = 0; b < 16; b++)
            slots.push_back(tp.add(Sblk(cr, i, b / 4, b % 4), Wblk(cL[k], i, b % 4, b / 4), (float)G5[b / 4], 0.f, 1));
        for (int b = 0; b < 16; b++) {
          if (iso != 0) {
            slots.push_back(-1);
            continue;
          }
          // Tr[F_{s1 s3} G_{s3 s1}], F = Phi3 Pm(P1), G = Phi4 Pm(P2)
          const int s1 = b / 4, s3 = b % 4, qf1 = iw[q[0]], qf2 = iw[q[1]];
          const double2* Fb = bF[i][qf1] + ((size_t)b * FK[qf1].size() + fpos[2 * k]) * N2;
          const double2* Gb = bF[i][qf2] + ((size_t)(s3 * 4 + s1) * FK[qf2].size() + fpos[2 * k + 1]) * N2;
          slots.push_back(tp.add(Fb, Gb, 1.f, 0.f, 1));
        }
        for (int h = 0; h < 4; h++)
          for (int b = 0; b < 16; b++) slots.push_back(b < ntw ? tws[twin[4 * k + h] * ntw + b] : -1);
        ent.push_back(k * npairs + pb.ent[i]);
        terms.insert(terms.end(), {i, cL[k] * Nt + pb.tf[i], cSq[k] * Nt + pb.ti[i], cDt[k] * Nt + pb.ti[i]});
      }
    }
    for (size_t k = 0; k < tp.tt.size(); k++) {
      tp.tt[k].out = trv + k;
      if (tra) tp.tt[k].absout = tra + k;
    }
    CTR_TRY(run_traces(c, tp.tt));
    void* d[4];
    CTR_TRY(upload_group(WS_MISC,
                         {{slots.data(), slots.size() * sizeof(int)},
                          {ent.data(), ent.size() * sizeof(int)},
                          {terms.data(), terms.size() * sizeof(int)},
                          {pb.T.data(), pb.T.size() * sizeof(const double2*)}},
                         d, s));
    if (rf.on) CTR_TRY(launch_block_norms((const double2* const*)d[3], np, 16, N, nT, s));
    {
      TimedLaunch tl(s, "pipi_combine");
      const int nitem = (int)ent.size();
      pipi_combine_sets_kernel<<<(nitem + 127) / 128, 128, 0, s>>>(trv, tra, (const int*)d[0], (const int*)d[1], nitem,
                                                                   iso, (double2*)corr, rf.eps_over_tol, rf.count,
                                                                   rf.list, (const int*)d[2], nT, nM, 1.0 / N);
      CTR_CUDA(cudaGetLastError());
    }
  }
  std::vector<int32_t> set_copy(sets, sets + 4 * nset);
  std::vector<Elem> elc(el);
  return refine_end(c, rf, 5, WS_REFINE, (double2*)corr,
                    [=](const std::vector<int>& units, double2* out, cudaStream_t ls) -> int {
                      // units = set * npairs + pair, ascending: one FP64 rerun per set
                      size_t u0 = 0;
                      while (u0 < units.size()) {
                        const int k = units[u0] / npairs;
                        size_t u1 = u0;
                        std::vector<int> pl;
                        while (u1 < units.size() && units[u1] / npairs == k) pl.push_back(units[u1++] % npairs);
                        CTR_TRY(pipi_core(N, Nt, tf_begin, tf_end, iso, prop_rows, prop_diag, elc, 1,
                                          set_copy.data() + 4 * k, (double*)(out + u0 * 5), ls, CTR_ENGINE_FP64, false,
                                          &pl));
                        u0 = u1;
                      }
                      return CTR_OK;
                    });
}

// --------------------------------------- rho -> pi pi and sigma -> pi pi over sets
// Both families contract X = T G R, R(t) = Phi_P2(t) taud(t) Phi_P1(t), with the
// sink operators: rho -> pi pi (lib/calculate_rhopi_core.h) takes Phi^{P1P2}_ip(tf)
// X_{s5 s2} for ip in {0, 1, 2 + idir}, the sigma -> pi pi triangle
// (lib/calculate_sigmapi_triangle_core.h) Phi^{x2}_ik(tf) X_b for ik in {0, 1}.
// Per set and pair, X is computed once and multiplied by all the sink operators
// the requested outputs need in one grid (slab = operator, right block = X
// block); the horizontal fish (lib/calculate_sigmapi_hor_fish_core.h) traces R
// against taud per time slice.

namespace {

// Row sums of batch items: row r of item it is trace slot itembase[it] + rowoff[r],
// conjugated where conj is set, times rcoef[r] where given; output o sums rows
// idx[off[o] .. off[o+1]) in that order into out[ent[it] * nout + o]; with trabs,
// entries whose error estimate exceeds the tolerance append ent * nout + o to the
// refinement list.
__global__ void rowsum_items_kernel(const double2* __restrict__ trv, const double* __restrict__ trabs,
                                    const int* __restrict__ itembase, const int* __restrict__ rowoff, int conj,
                                    const int* __restrict__ off, const int* __restrict__ idx,
                                    const float2* __restrict__ rcoef, int nout, const int* __restrict__ ent, int nitem,
                                    double2* __restrict__ out, double eps_over_tol, int* __restrict__ count,
                                    int* __restrict__ list) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nitem * nout) return;
  const int it = g / nout, o = g % nout, base = itembase[it];
  double re = 0.0, im = 0.0, sc = 0.0;
  for (int k = off[o]; k < off[o + 1]; k++) {
    const int r = idx[k], j = base + rowoff[r];
    double2 v = trv[j];
    if (conj) v.y = -v.y;
    double a = trabs ? trabs[j] : 0.0;
    if (rcoef) {  // the row's coefficient, applied as the trace kernel applies it
      const double2 c = make_double2((double)rcoef[r].x, (double)rcoef[r].y);
      v = cmul(c, v);
      a = sqrt(c.x * c.x + c.y * c.y) * a;
    }
    re += v.x;
    im += v.y;
    sc += a;
  }
  const size_t e = (size_t)ent[it] * nout + o;
  out[e] = make_double2(re, im);
  const double mag = sqrt(re * re + im * im);
  if (trabs && eps_over_tol > 0.0 && (!(sc * eps_over_tol <= mag) || (sc == 0.0 && mag > 0.0)))
    list[atomicAdd(count, 1)] = (int)e;
}

// Item tables of one row-sum launch (host), and their device copies.
struct RowItems {
  std::vector<int> base, ent;  // per item
  std::vector<int> off, csr;   // per row; rows of each output
  std::vector<float2> coef;    // per row, or empty
  int nout = 0, conj = 0;
  const int *d_base = nullptr, *d_off = nullptr, *d_csr = nullptr, *d_ent = nullptr;
  const float2* d_coef = nullptr;
};

// Uploads the tables of several row-sum launches in one staging copy.
int upload_items(const Ctx& c, std::vector<RowItems*> items) {
  std::vector<std::pair<const void*, size_t>> parts;
  for (RowItems* r : items) {
    parts.push_back({r->base.data(), r->base.size() * sizeof(int)});
    parts.push_back({r->off.data(), r->off.size() * sizeof(int)});
    parts.push_back({r->csr.data(), r->csr.size() * sizeof(int)});
    parts.push_back({r->ent.data(), r->ent.size() * sizeof(int)});
    parts.push_back({r->coef.data(), r->coef.size() * sizeof(float2)});
  }
  std::vector<void*> d(parts.size());
  CTR_TRY(upload_group(WS_MISC, parts, d.data(), c.s));
  for (size_t i = 0; i < items.size(); i++) {
    items[i]->d_base = (const int*)d[5 * i];
    items[i]->d_off = (const int*)d[5 * i + 1];
    items[i]->d_csr = (const int*)d[5 * i + 2];
    items[i]->d_ent = (const int*)d[5 * i + 3];
    items[i]->d_coef = items[i]->coef.empty() ? nullptr : (const float2*)d[5 * i + 4];
  }
  return CTR_OK;
}

int rowsum_items(const Ctx& c, const double2* trv, const double* tra, const RowItems& r, double2* out,
                 const Refine& rf) {
  if (r.ent.empty()) return CTR_OK;
  TimedLaunch tl(c.s, "rowsum_items");
  const int n = (int)r.ent.size() * r.nout;
  rowsum_items_kernel<<<(n + 127) / 128, 128, 0, c.s>>>(trv, rf.on ? tra : nullptr, r.d_base, r.d_off, r.conj, r.d_csr,
                                                        r.d_csr + r.nout + 1, r.d_coef, r.nout, r.d_ent,
                                                        (int)r.ent.size(), out, rf.eps_over_tol, rf.count, rf.list);
  CTR_CUDA(cudaGetLastError());
  return CTR_OK;
}

// ---- sink form of the rho -> pi pi and triangle traces
// A vertex is one output's sink side: operator `slab`, and for each spin s3 of the
// closing tau the spin s5 its gamma structure leads to, with coefficient c (g5(s3)
// included).  The output sum_{s2,s3} c(s3) Tr-Had(Op X_{s5 s2}, tau_{s3 s2}) with
// X = T G R is
//   sum_{s1,s2} g5(s1) Tr[Q_{s2 s1} R_{s1 s2}],
//   (Q_{s2 s1})^dag = H_{s1 s2} = sum_{s3} conj(c(s3)) (Op tau_{s5 s1})^dag tau_{s3 s2},
// where H does not depend on the momentum set: its products replace the 64 of X
// per set, and its traces against R, sum_b g5 conj(Tr-Had(H_b, R_b)), are all the
// entries of one Gram product (rows: pairs of a t_src x vertices; columns: sets).
struct Vertex {
  int slab, s5[4];
  float cre[4], cim[4];
};
struct SinkTerm {  // H = sum_k w_k (Op tau_{s5_k s1})^dag tau_{s3_k s2}
  int slab, n, s3[4], s5[4];
  float w[4];
};
struct SinkPlan {
  std::vector<SinkTerm> H;
  std::vector<std::vector<int>> stacks;                     // terms with the same s3 and w: one grid
  std::vector<std::vector<std::pair<int, float2>>> rows;    // vertex -> (term, coefficient)
  int products = 0;                                         // block products of the terms, per pair
};

// A term's blocks H_{s1 s2} may cancel in their sum over s3, and their norms, the scales of
// the Gram product's rows, with them: each row's scale is at least what the sum has
// without cancellation, (sum_k |Op tau_{s5_k s1}|^2 |tau_{s3_k s2}|^2 / Nev)^(1/2) for H_{s1 s2}
// against |R_{s1 s2}|.  0.78 takes the two factors' norms of |Re| + |Im| to a product's,
// so that the two scales agree where nothing cancels.  One CTA a (pair, term).
__global__ void __launch_bounds__(32) sink_scale_kernel(const SinkTerm* __restrict__ terms, int nH, int nops, int nC,
                                                        int Nt, double per_nev, const double* __restrict__ nO,
                                                        const double* __restrict__ nT, const double* __restrict__ nR,
                                                        const int* __restrict__ ti, double* __restrict__ tra) {
  __shared__ double est[16];
  const int i = blockIdx.x / nH;
  if (threadIdx.x < 16) {
    const SinkTerm& T = terms[blockIdx.x - i * nH];
    const int s1 = threadIdx.x / 4, s2 = threadIdx.x & 3;
    double a[4], m = 0.0, e = 0.0;
    for (int k = 0; k < T.n; k++) {
      a[k] = nO[((size_t)i * 16 + T.s5[k] * 4 + s1) * nops + T.slab] * nT[(size_t)i * 16 + T.s3[k] * 4 + s2];
      m = fmax(m, a[k]);
    }
    for (int k = 0; k < T.n && m > 0.0; k++) e += (a[k] / m) * (a[k] / m);
    est[threadIdx.x] = 0.78 * m * sqrt(e * per_nev);
  }
  __syncwarp();
  for (int ci = threadIdx.x; ci < nC; ci += 32) {
    double a = 0.0;
    for (int b = 0; b < 16; b++) a += est[b] * nR[((size_t)ci * Nt + ti[i]) * 16 + b];
    double& t = tra[(size_t)blockIdx.x * nC + ci];
    t = fmax(t, a);
  }
}

// False where a vertex's coefficients are not +-1 times one of them.  Two vertices
// of one operator that differ in the sign of half their spins (gamma_x and gamma_y)
// share two terms of two spins each, a and b: one is a + b, the other a - b.
bool sink_plan(const std::vector<Vertex>& V, SinkPlan& P) {
  std::vector<std::array<int, 4>> sg(V.size());
  std::map<std::array<int, 5>, std::vector<int>> by;
  P.rows.resize(V.size());
  for (size_t v = 0; v < V.size(); v++) {
    const Vertex& x = V[v];
    const float n0 = x.cre[0] * x.cre[0] + x.cim[0] * x.cim[0];
    for (int k = 0; k < 4; k++) {
      const float re = x.cre[k] * x.cre[0] + x.cim[k] * x.cim[0], im = x.cim[k] * x.cre[0] - x.cre[k] * x.cim[0];
      if (n0 == 0.f || im != 0.f || (re != n0 && re != -n0)) return false;
      sg[v][k] = re == n0 ? 1 : -1;
    }
    by[{x.slab, x.s5[0], x.s5[1], x.s5[2], x.s5[3]}].push_back((int)v);
  }
  auto term = [&](const Vertex& x, const std::array<int, 4>& s, const std::vector<int>& spins) {
    SinkTerm t;
    std::memset(&t, 0, sizeof(t));
    t.slab = x.slab;
    for (int k : spins) {
      t.s3[t.n] = k;
      t.s5[t.n] = x.s5[k];
      t.w[t.n++] = (float)s[k];
    }
    P.H.push_back(t);
    P.products += 16 * t.n;
    return (int)P.H.size() - 1;
  };
  for (auto& g : by) {
    std::map<std::array<int, 4>, std::vector<int>> sig;
    for (int v : g.second) sig[sg[v]].push_back(v);
    if (sig.size() == 2) {
      const auto &s1 = sig.begin()->first, &s2 = std::next(sig.begin())->first;
      std::vector<int> same, diff;
      for (int k = 0; k < 4; k++) (s1[k] == s2[k] ? same : diff).push_back(k);
      if (same.size() == 2) {
        const int a = term(V[g.second[0]], s1, same), b = term(V[g.second[0]], s1, diff);
        for (auto& e : sig)
          for (int v : e.second) {
            const float sb = e.first == s1 ? 1.f : -1.f;
            P.rows[v].push_back({a, make_float2(V[v].cre[0], V[v].cim[0])});
            P.rows[v].push_back({b, make_float2(sb * V[v].cre[0], sb * V[v].cim[0])});
          }
        continue;
      }
    }
    for (auto& e : sig) {
      const int h = term(V[e.second[0]], e.first, {0, 1, 2, 3});
      for (int v : e.second) P.rows[v].push_back({h, make_float2(V[v].cre[0], V[v].cim[0])});
    }
  }
  std::map<std::vector<int>, std::vector<int>> st;
  for (size_t h = 0; h < P.H.size(); h++) {
    std::vector<int> key;
    for (int k = 0; k < P.H[h].n; k++) {
      key.push_back(P.H[h].s3[k]);
      key.push_back(P.H[h].w[k] > 0.f ? 1 : -1);
    }
    st[key].push_back((int)h);
  }
  for (auto& e : st) P.stacks.push_back(e.second);
  return true;
}

}  // namespace

// rho -> pi pi for the polarisations idirs (rhopi [nset][idirs][pairs][4]), the
// sigma -> pi pi triangle (tri [nset][pairs][2]) and the horizontal fish (hor_fish
// [nset][Nt], or the listed time slices) of every set (P1, P2) = el[sets[2k ..]];
// with plist, the listed pairs only, in the list's order.  Row forms:
// lib/calculate_rhopi_core.h: coef * Tr[Phi_ip(tf) tau_{s5s6} Phi_P2(ti)
// taud(ti)_{s1s2} Phi_P1(ti) tau_{s3s2}^dag] with s6 = s1, s4 = s3 and coef =
// c(iop, s3, s5) g5(s1), so the sum over s1 is (T G R)_{s5 s2}; the triangle's
// sum over s3 is (T G R)_{s1 s5} alike.  sets_call: the closing traces may run as
// Gram products (split engine), and the batches take the sets' budget.
int rhopi_sigmapi_core(int N, int Nt, int tf_begin, int tf_end, const double* prop_rows, const double* prop_diag,
                       const std::vector<Elem>& el, const double* mom5, const double* mom2, int nset,
                       const int32_t* sets, const std::vector<int>& idirs, double* rhopi, double* tri,
                       double* hor_fish, cudaStream_t s, int engine, bool sets_call, const std::vector<int>* plist,
                       const std::vector<int>* tlist) {
  Ctx c{N, Nt, (size_t)N * N, s, engine};
  const bool rerun = plist || tlist;
  if (engine == CTR_ENGINE_SPLIT && !rerun) g_refined_last = 0;
  const size_t N2 = c.N2, blk16 = 16 * N2;
  const double2 *tau = (const double2*)prop_rows, *diag = (const double2*)prop_diag, *P5 = (const double2*)mom5,
                *P2x = (const double2*)mom2;
  const int rows = tf_end - tf_begin, nd = (int)idirs.size();
  const int npairs = rhopi || tri ? (plist ? (int)plist->size() : rows * Nt) : 0;
  const int nts = hor_fish ? (tlist ? (int)tlist->size() : Nt) : 0;
  const Tables& Tb = tables();
  // R(t) = Phi_P2 taud Phi_P1 for every set's (P2, P1)
  Combos cb(Nt);
  std::vector<int> cR(nset);
  for (int k = 0; k < nset; k++) {
    cR[k] = cb.use(sets[2 * k + 1], sets[2 * k]);
    for (int i = 0; i < npairs; i++) cb.need[cR[k]][(plist ? (*plist)[i] : i) % Nt] = 1;
    for (int i = 0; i < nts; i++) cb.need[cR[k]][tlist ? (*tlist)[i] : i] = 1;
  }
  const int nC = (int)cb.list.size();
  std::vector<const double2*> M;
  // a recomputation keeps its own R, so that the caller's stays valid
  CTR_TRY(per_t_products(c, diag, blk16, el, rerun ? WS_RPHI : WS_PHI, cb.list, cb.need,
                         sets_call ? 0 : 16 * (2 * (size_t)Nt + 4), M));
  std::vector<int32_t> sc(sets, sets + 2 * nset);
  std::vector<Elem> elc(el);

  // ---- horizontal fish: per set and time slice, sum_ab coef * Tr-Had(R_ab, taud_ab)
  // (lib/calculate_sigmapi_hor_fish_core.h)
  if (hor_fish) {
    Refine rf;
    CTR_TRY(refine_begin(c, (size_t)nset * nts, WS_REFINE, rf));
    const size_t ntr = (size_t)nset * nts * 16;
    void *trm, *tra = nullptr;
    CTR_TRY(workspace(WS_ROWS).get(ntr * sizeof(double2), &trm));
    if (rf.on) CTR_TRY(workspace(WS_ROWABS).get(ntr * sizeof(double), &tra));
    std::vector<TraceTask> tt;
    tt.reserve(ntr);
    RowItems ri;
    ri.nout = 1;
    for (int k = 0; k < nset; k++)
      for (int i = 0; i < nts; i++) {
        const int t = tlist ? (*tlist)[i] : i;
        for (int b = 0; b < 16; b++) {
          const int ab = Tb.hf_spin[b][0] * 4 + Tb.hf_spin[b][1];
          tt.push_back(tr(M[(size_t)cR[k] * Nt + t] + ab * N2, diag + t * blk16 + ab * N2,
                          (double2*)trm + tt.size(), Tb.hf_coef[b][0], Tb.hf_coef[b][1], 0));
          if (tra) tt.back().absout = (double*)tra + (tt.size() - 1);
        }
        ri.base.push_back((int)tt.size() - 16);
        ri.ent.push_back(k * nts + i);
      }
    ri.csr = {0, 16};
    for (int b = 0; b < 16; b++) {
      ri.csr.push_back(b);
      ri.off.push_back(b);
    }
    CTR_TRY(run_traces(c, tt));
    CTR_TRY(upload_items(c, {&ri}));
    CTR_TRY(rowsum_items(c, (double2*)trm, (double*)tra, ri, (double2*)hor_fish, rf));
    CTR_TRY(refine_end(c, rf, 1, WS_REFINE, (double2*)hor_fish,
                       [=](const std::vector<int>& units, double2* out, cudaStream_t ls) -> int {
                         size_t u0 = 0;
                         while (u0 < units.size()) {  // units = set * Nt + t: one FP64 rerun per set
                           const int k = units[u0] / nts;
                           std::vector<int> tl;
                           size_t u1 = u0;
                           while (u1 < units.size() && units[u1] / nts == k) tl.push_back(units[u1++] % nts);
                           CTR_TRY(rhopi_sigmapi_core(N, Nt, tf_begin, tf_end, prop_rows, prop_diag, elc, mom5, mom2,
                                                      1, sc.data() + 2 * k, {}, nullptr, nullptr, (double*)(out + u0),
                                                      ls, CTR_ENGINE_FP64, false, nullptr, &tl));
                           u0 = u1;
                         }
                         return CTR_OK;
                       }));
  }
  if (!rhopi && !tri) return CTR_OK;

  // ---- sink operators of the grid: the rho operators the three polarisations use, then sigma's two
  struct Grp {
    int iop, s2, s3, s5, slab;
    float cre, cim;
  };
  std::vector<int> ops;  // slab -> operator: 0..4 rho (mom5), 5..6 sigma (mom2)
  std::vector<int> slab_of(7, -1);
  std::vector<std::vector<Grp>> grp(nd);
  std::vector<std::vector<int>> csr_rp(nd);
  if (rhopi)
    for (int d = 0; d < nd; d++) {
      const int idir = idirs[d];
      for (int bx = 0; bx < 256; bx++) {
        const int r = idir * 256 + bx;
        const int16_t* sp = Tb.rhopi_spin[r];
        const int s1 = sp[0];
        if (sp[5] != s1 || sp[3] != sp[2])
          return fail(CTR_ERR_ARG, "rho-pipi table row %d not gamma_5-diagonal", r);
        if (s1 != 0) continue;  // one representative per group (coef x g5(s1) sums over s1)
        const int ip = Tb.rhopi_ip[r];
        if (slab_of[ip] < 0) {
          slab_of[ip] = (int)ops.size();
          ops.push_back(ip);
        }
        grp[d].push_back(Grp{bx / 64, sp[1], sp[2], sp[4], slab_of[ip], Tb.rhopi_coef[r][0] * G5[s1],
                             Tb.rhopi_coef[r][1] * G5[s1]});
      }
      // CSR of the 4 operators over the groups, in group order
      std::vector<int> off(5, 0), idx(grp[d].size());
      for (auto& g : grp[d]) off[g.iop + 1]++;
      for (int o = 0; o < 4; o++) off[o + 1] += off[o];
      std::vector<int> fill(off.begin(), off.end() - 1);
      for (size_t g = 0; g < grp[d].size(); g++) idx[fill[grp[d][g].iop]++] = (int)g;
      csr_rp[d] = off;
      csr_rp[d].insert(csr_rp[d].end(), idx.begin(), idx.end());
    }
  if (tri)
    for (int ik = 0; ik < 2; ik++) {
      slab_of[5 + ik] = (int)ops.size();
      ops.push_back(5 + ik);
    }
  const int nops = (int)ops.size();
  // the distinct traces (slab, X block, Z block) of the polarisations' groups
  std::vector<std::tuple<int, int, int>> uniq;
  std::vector<std::vector<int>> uidx(nd);
  if (rhopi) {
    std::map<std::tuple<int, int, int>, int> at;
    for (int d = 0; d < nd; d++)
      for (const Grp& g : grp[d]) {
        const auto key = std::make_tuple(g.slab, g.s5 * 4 + g.s2, g.s3 * 4 + g.s2);
        auto it = at.find(key);
        if (it == at.end()) {
          it = at.emplace(key, (int)uniq.size()).first;
          uniq.push_back(key);
        }
        uidx[d].push_back(it->second);
      }
  }
  std::vector<int> csr_tr = {0, 16, 32};
  for (int k = 0; k < 32; k++) csr_tr.push_back(k);

  const size_t blk_pair = 16 * ((size_t)nC + nops);
  const size_t tr_pair = (size_t)nset * (uniq.size() + (tri ? 32 : 0));
  const size_t per_pair = blk_pair * N2 * sizeof(double2) + tr_pair * (sizeof(double2) + sizeof(double));
  const size_t budget = sets_call ? sets_budget() : CHAIN_BUDGET;
  const int batch = std::max(1, std::min(npairs, (int)(budget / std::max<size_t>(per_pair, 1))));
  // closing-trace form on the split engine (chains.trace_form): when it is known
  // to be the Gram products, the FP64 trace tasks are not built
  const std::string trace_shape =
      "nev=" + std::to_string(N) + ",m=" + std::to_string(4 * nC) + ",n=" + std::to_string(4 * nops);
  int known_form = 0;
  const bool gram = c.engine == CTR_ENGINE_SPLIT && sets_call;
  const bool fp64_traces_needed = !gram ||
                                  !tune_peek("chains.trace_form", trace_shape, 2, 1, &known_form) || known_form == 0;
  Refine rf_rp, rf_tr;
  if (rhopi) CTR_TRY(refine_begin(c, (size_t)nset * nd * npairs * 4, WS_REFINE, rf_rp));
  if (tri) CTR_TRY(refine_begin(c, (size_t)nset * npairs * 2, WS_SPLITJOBS3, rf_tr));
  // The sink form takes its place where it costs less.  In block products a pair: the
  // terms' products, a quarter dearer each (two terms of K, four columns of blocks), instead
  // of 64 a set, and 10.4 for each row of 16 blocks that a Gram product has, its tiles of
  // 128 rows and 48 columns counted whole (0.65 of a block product a block's slices and its
  // share of that product): nH rows a sink time of a batch and a column a set, once a
  // t_src, against a row a set and a column an operator.  At least 11 sets with every
  // output, 9 for rho -> pi pi and 2 for the triangle, where the tiles are full.  Measured
  // (Nev = 128, Lt = 32, ms, with X / sink form): 8 sink times, 11 and 27 sets, every output
  // 72 / 70 and 137 / 75, triangle 65 / 25 and 130 / 31; 4 sink times, every output 38 / 41
  // and 74 / 47, triangle of 2 and 3 sets 15.7 / 16.4 and 18.2 / 16.8; one sink time,
  // triangle of 2, 16 and 27 sets 4.8 / 12.4, 16.1 / 17.0 and 25.1 / 21.1.
  SinkPlan sp;
  bool sink = gram && !fp64_traces_needed;
  if (sink) {
    std::vector<Vertex> V;
    for (int d = 0; d < nd && rhopi; d++)
      for (int iop = 0; iop < 4; iop++) {
        Vertex v;
        std::memset(&v, 0, sizeof(v));
        for (const Grp& g : grp[d])
          if (g.iop == iop && g.s2 == 0) {
            v.slab = g.slab;
            v.s5[g.s3] = g.s5;
            v.cre[g.s3] = g.cre;
            v.cim[g.s3] = g.cim;
          }
        V.push_back(v);
      }
    for (int ik = 0; ik < 2 && tri; ik++)
      V.push_back(Vertex{slab_of[5 + ik], {0, 1, 2, 3}, {(float)G5[0], (float)G5[1], (float)G5[2], (float)G5[3]}, {}});
    sink = sink_plan(V, sp) && sp.products + 10.4 * sp.H.size() < 64.0 * nC + 10.4 * (nC + nops);
  }
  const int nH = (int)sp.H.size();
  // sink times a batch: their rows fill two tiles of a t_src's Gram product
  const int hmax = std::max(1, 256 / std::max(1, nH));
  if (sink) {
    auto tiles = [](int n, int size) { return (double)((n + size - 1) / size * size); };
    const int h = std::min(rows, hmax);
    const double rows_sink = (tiles(h * nH, 128) + tiles(nC, 48)) / h;
    const double rows_x = (tiles(4 * nC, 128) + tiles(4 * nops, 48)) / 4;  // four products a pair, of 4 of the 16 blocks
    sink = 1.25 * sp.products + 10.4 * rows_sink < 64.0 * nC + 10.4 * rows_x;
  }
  const size_t per_pair_sink = 16 * ((size_t)nops + nH) * N2 * sizeof(double2) +
                               (size_t)nH * nC * (sizeof(double2) + sizeof(double));
  const int batch_sink = std::max(1, std::min(npairs, (int)(budget / per_pair_sink)));
  // norms of R (for the call), of Op tau and of tau (for a batch)
  const bool scales = sink && (rf_rp.on || rf_tr.on);
  double *nR = nullptr, *nO = nullptr, *nT = nullptr;
  if (scales) {
    void* p;
    CTR_TRY(workspace(WS_NORMS).get(16 * ((size_t)nC * Nt + (size_t)batch_sink * (nops + 1)) * sizeof(double), &p));
    nR = (double*)p;
    nO = nR + (size_t)16 * nC * Nt;
    nT = nO + (size_t)16 * batch_sink * nops;
    void* d;
    CTR_TRY(upload(WS_MISC, M.data(), M.size() * sizeof(const double2*), &d, c.s));
    CTR_TRY(launch_block_norms((const double2* const*)d, nC * Nt, 16, N, nR, c.s));
  }
  for (const PairBatch& pb : sink ? pair_batches(tau, blk16, Nt, tf_begin, rows, batch_sink, plist, hmax)
                                  : std::vector<PairBatch>()) {
    const int np = (int)pb.ent.size(), ng = (int)pb.by_ti.size();
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get((size_t)np * per_pair_sink, &mem));
    double2* bO = (double2*)mem;                      // Op(tf) tau_b, block (b, slab) of pair i
    double2* bH = bO + (size_t)np * 16 * nops * N2;   // terms, by stack
    double2* trv = bH + (size_t)np * 16 * nH * N2;
    double* tra = (rf_rp.on || rf_tr.on) ? (double*)(trv + (size_t)np * nH * nC) : nullptr;
    auto Oblk = [&](int sl, int i, int b) { return bO + ((size_t)i * 16 * nops + (size_t)b * nops + sl) * N2; };
    std::vector<GridTask> g0, g1;
    std::vector<const double2*> hblk((size_t)np * nH * 16);  // [pair][term][s1 * 4 + s2]
    for (int i = 0; i < np; i++) {
      for (int jb = 0; jb < 2; jb++) {
        GridTask go = make_grid(nops, 8, 1, kOne, 0, 0);
        for (int sl = 0; sl < nops; sl++)
          go.A[sl] = ops[sl] < 5 ? P5 + ((size_t)pb.tf[i] * 5 + ops[sl]) * N2
                                 : P2x + ((size_t)pb.tf[i] * 2 + ops[sl] - 5) * N2;
        for (int j = 0; j < 8; j++) {
          go.B[j][0] = pb.T[i] + (size_t)(8 * jb + j) * N2;
          go.C0[j] = Oblk(0, i, 8 * jb + j);
        }
        g0.push_back(std::move(go));
      }
      double2* next = bH + (size_t)i * 16 * nH * N2;
      for (const std::vector<int>& st : sp.stacks) {
        // slab (term, s1), right block s2
        const SinkTerm& t0 = sp.H[st[0]];
        const int m = (int)st.size();
        GridTask gh = make_grid(4 * m, 4, t0.n, t0.w, (1 << t0.n) - 1, 0);
        for (int u = 0; u < m; u++)
          for (int s1 = 0; s1 < 4; s1++)
            for (int k = 0; k < t0.n; k++) {
              const SinkTerm& t = sp.H[st[u]];
              gh.A[(size_t)(u * 4 + s1) * t0.n + k] = Oblk(t.slab, i, t.s5[k] * 4 + s1);
            }
        for (int j = 0; j < 4; j++) {
          for (int k = 0; k < t0.n; k++) gh.B[j][k] = pb.T[i] + (size_t)(t0.s3[k] * 4 + j) * N2;
          gh.C0[j] = next + (size_t)j * 4 * m * N2;
        }
        for (int u = 0; u < m; u++)
          for (int b = 0; b < 16; b++)
            hblk[((size_t)i * nH + st[u]) * 16 + b] = next + ((size_t)(b % 4) * 4 * m + u * 4 + b / 4) * N2;
        next += (size_t)16 * m * N2;
        g1.push_back(std::move(gh));
      }
    }
    CTR_TRY(run_grids(c, g0, WS_TASKS));
    CTR_TRY(run_grids(c, g1, WS_TASKS2));
    GramRows gr;
    size_t maxm = 0;
    for (auto& v : pb.by_ti) maxm = std::max(maxm, v.size());
    gr.ngroup = ng;
    gr.nblk = 16;
    gr.mrows = (int)maxm * nH;
    gr.ncols = nC;
    for (int b = 0; b < 16; b++)
      if (G5[b / 4] < 0) gr.negative |= 1u << b;
    gr.left.assign((size_t)ng * 16 * gr.mrows, nullptr);
    gr.right.resize((size_t)ng * 16 * nC);
    gr.rowbase.assign((size_t)ng * gr.mrows, -1);
    for (int g = 0; g < ng; g++) {
      const std::vector<int>& mem_i = pb.by_ti[g];
      for (size_t pp = 0; pp < mem_i.size(); pp++)
        for (int h = 0; h < nH; h++) {
          gr.rowbase[(size_t)g * gr.mrows + pp * nH + h] = (mem_i[pp] * nH + h) * nC;
          for (int b = 0; b < 16; b++)
            gr.left[((size_t)g * 16 + b) * gr.mrows + pp * nH + h] = hblk[((size_t)mem_i[pp] * nH + h) * 16 + b];
        }
      for (int b = 0; b < 16; b++)
        for (int ci = 0; ci < nC; ci++)
          gr.right[((size_t)g * 16 + b) * nC + ci] = M[(size_t)ci * Nt + pb.ti[mem_i[0]]] + (size_t)b * N2;
    }
    std::vector<RowItems> it(nd + 1);  // polarisations, then the triangle
    size_t v0 = 0;
    for (int d = 0; d <= nd; d++) {
      RowItems& r = it[d];
      if (d < nd ? !rhopi : !tri) continue;
      r.nout = d < nd ? 4 : 2;
      r.conj = 1;
      r.csr.push_back(0);
      for (int o = 0; o < r.nout; o++, v0++) {
        for (auto& e : sp.rows[v0]) {
          r.off.push_back(e.first * nC);
          r.coef.push_back(e.second);
        }
        r.csr.push_back((int)r.off.size());
      }
      for (size_t k = 0; k < r.off.size(); k++) r.csr.push_back((int)k);
      for (int i = 0; i < np; i++)
        for (int k = 0; k < nset; k++) {
          r.base.push_back(i * nH * nC + cR[k]);
          r.ent.push_back((d < nd ? k * nd + d : k) * npairs + pb.ent[i]);
        }
    }
    CTR_TRY(gram_rows(N, gr, trv, tra, c.s));
    if (scales) {
      std::vector<const double2*> bases;
      for (int i = 0; i < np; i++) bases.push_back(Oblk(0, i, 0));
      bases.insert(bases.end(), pb.T.begin(), pb.T.end());
      void* d[3];
      CTR_TRY(upload_group(WS_ROWTASKS,
                           {{bases.data(), bases.size() * sizeof(const double2*)},
                            {sp.H.data(), sp.H.size() * sizeof(SinkTerm)},
                            {pb.ti.data(), pb.ti.size() * sizeof(int)}},
                           d, c.s));
      CTR_TRY(launch_block_norms((const double2* const*)d[0], np, 16 * nops, N, nO, c.s));
      CTR_TRY(launch_block_norms((const double2* const*)d[0] + np, np, 16, N, nT, c.s));
      TimedLaunch tl(c.s, "sink_scale");
      sink_scale_kernel<<<np * nH, 32, 0, c.s>>>((const SinkTerm*)d[1], nH, nops, nC, Nt, 1.0 / N, nO, nT, nR,
                                                 (const int*)d[2], tra);
      CTR_CUDA(cudaGetLastError());
    }
    std::vector<RowItems*> items;
    for (RowItems& r : it) items.push_back(&r);
    CTR_TRY(upload_items(c, items));
    for (int d = 0; d < nd; d++) CTR_TRY(rowsum_items(c, trv, tra, it[d], (double2*)rhopi, rf_rp));
    CTR_TRY(rowsum_items(c, trv, tra, it[nd], (double2*)tri, rf_tr));
  }
  for (const PairBatch& pb : sink ? std::vector<PairBatch>()
                                  : pair_batches(tau, blk16, Nt, tf_begin, rows, batch, plist)) {
    const int np = (int)pb.ent.size(), ng = (int)pb.by_ti.size();
    void* mem;
    CTR_TRY(workspace(WS_SCRATCH).get((size_t)np * per_pair, &mem));
    double2* base = (double2*)mem;
    size_t used = 0;
    auto alloc = [&](size_t nblk) {
      double2* p = base + used;
      used += nblk * N2;
      return p;
    };
    std::vector<double2*> bX((size_t)ng * nC), bZ(np);
    for (int g = 0; g < ng; g++)
      for (int ci = 0; ci < nC; ci++) bX[(size_t)g * nC + ci] = alloc(16 * pb.by_ti[g].size());
    for (int i = 0; i < np; i++) bZ[i] = alloc(16 * (size_t)nops);
    // X(ci, i)_{a b} and Z(op slab, i)_b = Op(tf)^dag tau_b (shared by all sets)
    auto Xblk = [&](int ci, int i, int a, int b) {
      const int g = pb.gti[i];
      return bX[(size_t)g * nC + ci] + ((size_t)b * 4 * pb.by_ti[g].size() + pb.pti[i] * 4 + a) * N2;
    };
    auto Zblk = [&](int sl, int i, int b) { return bZ[i] + ((size_t)b * nops + sl) * N2; };
    std::vector<GridTask> g0;
    for (int g = 0; g < ng; g++) {
      const std::vector<int>& mem_i = pb.by_ti[g];
      const int m = (int)mem_i.size(), ti = pb.ti[mem_i[0]];
      for (int c0 = 0; c0 < nC; c0 += 2) {
        // X = T G R: slab (pair, row block a), right block b of up to two R(t_src)
        const int nf = std::min(2, nC - c0);
        GridTask gx = make_grid(4 * m, 4 * nf, 4, kG5, 0, 0);
        for (int pp = 0; pp < m; pp++)
          for (int a = 0; a < 4; a++)
            for (int kk = 0; kk < 4; kk++)
              gx.A[(size_t)(pp * 4 + a) * 4 + kk] = pb.T[mem_i[pp]] + (size_t)(a * 4 + kk) * N2;
        for (int u = 0; u < nf; u++)
          for (int j = 0; j < 4; j++) {
            for (int kk = 0; kk < 4; kk++)
              gx.B[u * 4 + j][kk] = M[(size_t)(c0 + u) * Nt + ti] + (size_t)(kk * 4 + j) * N2;
            gx.C0[u * 4 + j] = bX[(size_t)g * nC + c0 + u] + (size_t)j * 4 * m * N2;
          }
        g0.push_back(std::move(gx));
      }
    }
    for (int i = 0; i < np; i++)
      for (int jb = 0; jb < 2; jb++) {
        // Z = Op(tf)^dag tau_b: slab = sink operator, right block b of tau
        GridTask gz = make_grid(nops, 8, 1, kOne, 1, 0);
        for (int sl = 0; sl < nops; sl++)
          gz.A[sl] = ops[sl] < 5 ? P5 + ((size_t)pb.tf[i] * 5 + ops[sl]) * N2
                                 : P2x + ((size_t)pb.tf[i] * 2 + ops[sl] - 5) * N2;
        for (int j = 0; j < 8; j++) {
          const int b = 8 * jb + j;
          gz.B[j][0] = pb.T[i] + (size_t)b * N2;
          gz.C0[j] = bZ[i] + (size_t)b * nops * N2;
        }
        g0.push_back(std::move(gz));
      }
    CTR_TRY(run_grids(c, g0, WS_TASKS));  // while the host lists the traces
    // traces
    const size_t ntr = (size_t)np * tr_pair;
    double2* trv = base + used;
    double* tra = (rf_rp.on || rf_tr.on) ? (double*)(trv + ntr) : nullptr;
    if (used * sizeof(double2) + ntr * (sizeof(double2) + sizeof(double)) > (size_t)np * per_pair)
      return fail(CTR_ERR_ALLOC, "ctr_rhopi_sigmapi_sets: batch arena overflow");
    TracePlan tp;
    tp.keep = fp64_traces_needed;
    if (tp.keep) tp.tt.reserve((size_t)np * tr_pair);
    // on the split engine the same traces as Gram products: group i * 4 + s2 of
    // pair i pairs the X blocks (set combination ci, row block s5, column block
    // s2) with the Z blocks (sink operator slab, tau block (s3, s2)); every trace
    // takes an X and a Z block with the same s2
    GramPlan gp;
    if (gram) {
      gp.tr.reserve((size_t)np * tr_pair);
      gp.ngroup = 4 * np;
      gp.group_run = 4;  // a pair's traces interleave its four s2 groups
      gp.mrows = 4 * nC;
      gp.ncols = 4 * nops;
      gp.left.resize((size_t)gp.ngroup * gp.mrows);
      gp.right.resize((size_t)gp.ngroup * gp.ncols);
      for (int i = 0; i < np; i++)
        for (int s2 = 0; s2 < 4; s2++) {
          const size_t g = (size_t)i * 4 + s2;
          for (int ci = 0; ci < nC; ci++)
            for (int s5 = 0; s5 < 4; s5++) gp.left[g * gp.mrows + ci * 4 + s5] = Xblk(ci, i, s5, s2);
          for (int sl = 0; sl < nops; sl++)
            for (int s3 = 0; s3 < 4; s3++) gp.right[g * gp.ncols + sl * 4 + s3] = Zblk(sl, i, s3 * 4 + s2);
        }
    }
    RowItems it_tr;
    std::vector<RowItems> it_rp(nd);
    for (int d = 0; d < nd && rhopi; d++) {
      it_rp[d].nout = 4;
      it_rp[d].csr = csr_rp[d];
      it_rp[d].off = uidx[d];
      for (const Grp& g : grp[d]) it_rp[d].coef.push_back(make_float2(g.cre, g.cim));
    }
    it_tr.nout = 2;
    it_tr.csr = csr_tr;
    for (int r = 0; r < 32; r++) it_tr.off.push_back(r);
    for (int i = 0; i < np; i++) {
      const int pair = pb.ent[i];
      for (int k = 0; k < nset; k++) {
        const int ci = cR[k];
        if (rhopi) {
          // Tr-Had(X_{s5 s2}, Phi_ip^dag tau_{s3 s2}) without its coefficient, once for the
          // polarisations (those of ip = 0, 1 are shared); the row sums apply the coefficients
          const int base = tp.n;
          for (const auto& u : uniq) {
            const int xb = std::get<1>(u), zb = std::get<2>(u);
            const int slot = tp.add(Xblk(ci, i, xb / 4, xb % 4), Zblk(std::get<0>(u), i, zb), 1.f, 0.f, 0);
            if (gram) gp.tr.push_back({i * 4 + xb % 4, ci * 4 + xb / 4, std::get<0>(u) * 4 + zb / 4, slot, 1.f, 0.f});
          }
          for (int d = 0; d < nd; d++) {
            it_rp[d].base.push_back(base);
            it_rp[d].ent.push_back((k * nd + d) * npairs + pair);
          }
        }
        if (tri) {
          it_tr.base.push_back(tp.n);
          for (int ik = 0; ik < 2; ik++)
            for (int b = 0; b < 16; b++) {
              const int slot = tp.add(Xblk(ci, i, b / 4, b % 4), Zblk(slab_of[5 + ik], i, b), (float)G5[b / 4], 0.f, 0);
              if (gram) gp.tr.push_back({i * 4 + b % 4, ci * 4 + b / 4, slab_of[5 + ik] * 4 + b / 4, slot, (float)G5[b / 4], 0.f});
            }
          it_tr.ent.push_back(k * npairs + pair);
        }
      }
    }
    for (size_t k = 0; k < tp.tt.size(); k++) {
      tp.tt[k].out = trv + k;
      if (tra) tp.tt[k].absout = tra + k;
    }
    if (gram) {
      // 0: the FP64 trace kernel, 1: Gram products on the tensor cores
      int form = 1;
      auto run = [&](int f) { return f ? trace_gram(N, gp, trv, tra, c.s) : run_traces(c, tp.tt); };
      CTR_TRY(tune_resolve("chains.trace_form", trace_shape, 2, 1, c.s, run, &form));
      if (form == 0 && !tp.keep) return fail(CTR_ERR_ARG, "chains.trace_form: FP64 traces chosen but not planned");
      CTR_TRY(run(form));
    } else {
      CTR_TRY(run_traces(c, tp.tt));
    }
    std::vector<RowItems*> items = {&it_tr};
    for (RowItems& r : it_rp) items.push_back(&r);
    CTR_TRY(upload_items(c, items));
    for (const RowItems& r : it_rp) CTR_TRY(rowsum_items(c, trv, tra, r, (double2*)rhopi, rf_rp));
    if (tri) CTR_TRY(rowsum_items(c, trv, tra, it_tr, (double2*)tri, rf_tr));
  }
  if (rhopi)
    CTR_TRY(refine_end(c, rf_rp, 4, WS_REFINE, (double2*)rhopi,
                       [=](const std::vector<int>& units, double2* out, cudaStream_t ls) -> int {
                         size_t u0 = 0;  // units = (set * nd + d) * npairs + pair
                         while (u0 < units.size()) {
                           const int kd = units[u0] / npairs;
                           std::vector<int> pl;
                           size_t u1 = u0;
                           while (u1 < units.size() && units[u1] / npairs == kd) pl.push_back(units[u1++] % npairs);
                           CTR_TRY(rhopi_sigmapi_core(N, Nt, tf_begin, tf_end, prop_rows, prop_diag, elc, mom5, mom2,
                                                      1, sc.data() + 2 * (kd / nd), {idirs[kd % nd]},
                                                      (double*)(out + u0 * 4), nullptr, nullptr, ls, CTR_ENGINE_FP64,
                                                      false, &pl, nullptr));
                           u0 = u1;
                         }
                         return CTR_OK;
                       }));
  if (tri)
    CTR_TRY(refine_end(c, rf_tr, 2, WS_SPLITJOBS3, (double2*)tri,
                       [=](const std::vector<int>& units, double2* out, cudaStream_t ls) -> int {
                         size_t u0 = 0;  // units = set * npairs + pair
                         while (u0 < units.size()) {
                           const int k = units[u0] / npairs;
                           std::vector<int> pl;
                           size_t u1 = u0;
                           while (u1 < units.size() && units[u1] / npairs == k) pl.push_back(units[u1++] % npairs);
                           CTR_TRY(rhopi_sigmapi_core(N, Nt, tf_begin, tf_end, prop_rows, prop_diag, elc, mom5, mom2,
                                                      1, sc.data() + 2 * k, {}, nullptr, (double*)(out + u0 * 2),
                                                      nullptr, ls, CTR_ENGINE_FP64, false, &pl, nullptr));
                           u0 = u1;
                         }
                         return CTR_OK;
                       }));
  return CTR_OK;
}

// -------------------------------------------------------------- loop unity
// lib/calculate_loop_unity_core.h: L(t) = sum_s Tr[taud(t)_{ss} Phi(t)] (trace of a product: Nev^2 work).
int loop_unity_fp64(int N, int Nt, const double* prop_diag, const double* mom, double* loop, cudaStream_t s) {
  return launch_loop_unity((const double2*)prop_diag, (const double2*)mom, N, Nt, (double2*)loop, s);
}

}  // namespace ctr

// ------------------------------------------------------------------ C ABI
static int chain_args(int engine, int nev, int nt, int tf_begin, int tf_end) {
  if (engine != CTR_ENGINE_FP64 && engine != CTR_ENGINE_SPLIT) return ctr::fail(CTR_ERR_ARG, "unknown engine %d", engine);
  if (nev < 1 || nt < 1 || tf_begin < 0 || tf_end > nt || tf_begin >= tf_end)
    return ctr::fail(CTR_ERR_ARG, "bad sizes (nev=%d nt=%d t_sink [%d,%d))", nev, nt, tf_begin, tf_end);
  return CTR_OK;
}

namespace ctr {

// One call's own elementals, [nt][nev][nev] each; set[k]: the first of them with
// the k-th one's address.
std::vector<Elem> elems(int nev, const std::vector<const double*>& p, int32_t* set) {
  std::vector<Elem> el;
  for (size_t k = 0; k < p.size(); k++) {
    size_t j = 0;
    while (j < el.size() && el[j].p != (const double2*)p[k]) j++;
    if (j == el.size()) el.push_back({(const double2*)p[k], (size_t)nev * nev});
    set[k] = (int32_t)j;
  }
  return el;
}

// The momenta of one [nt][nphi][nev][nev] array.
static std::vector<Elem> elems(int nev, const double* phi, int nphi) {
  std::vector<Elem> el(nphi);
  for (int q = 0; q < nphi; q++) el[q] = {(const double2*)phi + (size_t)q * nev * nev, (size_t)nphi * nev * nev};
  return el;
}

}  // namespace ctr

static bool aligned(const void* p) { return p && (((uintptr_t)p & 15) == 0); }

extern "C" {

int ctr_rhopi(int engine, int nev, int nt, int tf_begin, int tf_end, int idir, const double* prop_rows,
              const double* prop_diag, const double* mom_p1, const double* mom_p2, const double* mom5_p1p2,
              double* corr, void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, tf_begin, tf_end));
  if (!aligned(prop_rows) || !aligned(prop_diag) || !aligned(mom_p1) || !aligned(mom_p2) || !aligned(mom5_p1p2) ||
      !aligned(corr))
    return ctr::fail(CTR_ERR_ARG, "ctr_rhopi: null or misaligned pointer");
  if (idir < 0 || idir > 2) return ctr::fail(CTR_ERR_ARG, "idir %d not in {0,1,2}", idir);
  int32_t set[2];
  const std::vector<ctr::Elem> el = ctr::elems(nev, {mom_p1, mom_p2}, set);
  return ctr::rhopi_sigmapi_core(nev, nt, tf_begin, tf_end, prop_rows, prop_diag, el, mom5_p1p2, nullptr, 1, set,
                                 {idir}, corr, nullptr, nullptr, (cudaStream_t)stream, engine, false, nullptr,
                                 nullptr);
}

int ctr_pipi(int engine, int nev, int nt, int tf_begin, int tf_end, int isospin, const double* prop_rows,
             const double* prop_diag, const double* p1, const double* p2, const double* p3, const double* p4,
             double* corr, void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, tf_begin, tf_end));
  if (isospin != 0 && isospin != 1) return ctr::fail(CTR_ERR_ARG, "isospin must be 0 (I=0) or 1 (I=1)");
  if (!aligned(prop_rows) || !aligned(prop_diag) || !aligned(p1) || !aligned(p2) || !aligned(p3) || !aligned(p4) ||
      !aligned(corr))
    return ctr::fail(CTR_ERR_ARG, "ctr_pipi: null or misaligned pointer");
  int32_t set[4];
  const std::vector<ctr::Elem> el = ctr::elems(nev, {p1, p2, p3, p4}, set);
  return ctr::pipi_core(nev, nt, tf_begin, tf_end, isospin, prop_rows, prop_diag, el, 1, set, corr,
                        (cudaStream_t)stream, engine, false, nullptr);
}

int ctr_pipi_sets(int engine, int nev, int nt, int tf_begin, int tf_end, int isospin, const double* prop_rows,
                  const double* prop_diag, const double* phi, int nphi, int nset, const int32_t* sets, double* corr,
                  void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, tf_begin, tf_end));
  if (isospin != 0 && isospin != 1) return ctr::fail(CTR_ERR_ARG, "isospin must be 0 (I=0) or 1 (I=1)");
  if (nphi < 1 || nset < 1 || !sets) return ctr::fail(CTR_ERR_ARG, "ctr_pipi_sets: nphi=%d, nset=%d", nphi, nset);
  if (!aligned(prop_rows) || !aligned(prop_diag) || !aligned(phi) || !aligned(corr))
    return ctr::fail(CTR_ERR_ARG, "ctr_pipi_sets: null or misaligned pointer");
  for (int k = 0; k < 4 * nset; k++)
    if (sets[k] < 0 || sets[k] >= nphi)
      return ctr::fail(CTR_ERR_ARG, "ctr_pipi_sets: elemental index %d not in [0,%d)", sets[k], nphi);
  return ctr::pipi_core(nev, nt, tf_begin, tf_end, isospin, prop_rows, prop_diag, ctr::elems(nev, phi, nphi), nset,
                        sets, corr, (cudaStream_t)stream, engine, true, nullptr);
}

int ctr_rhopi_sigmapi_sets(int engine, int nev, int nt, int tf_begin, int tf_end, const double* prop_rows,
                           const double* prop_diag, const double* phi, int nphi, const double* mom5_p1p2,
                           const double* mom2_p1p2, int nset, const int32_t* sets, double* rhopi, double* triangle,
                           double* hor_fish, void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, tf_begin, tf_end));
  if (nphi < 1 || nset < 1 || !sets)
    return ctr::fail(CTR_ERR_ARG, "ctr_rhopi_sigmapi_sets: nphi=%d, nset=%d", nphi, nset);
  if (!aligned(prop_diag) || !aligned(phi) || ((rhopi || triangle) && !aligned(prop_rows)) ||
      (rhopi && (!aligned(mom5_p1p2) || !aligned(rhopi))) || ((triangle || hor_fish) && !aligned(mom2_p1p2)) ||
      (triangle && !aligned(triangle)) || (hor_fish && !aligned(hor_fish)))
    return ctr::fail(CTR_ERR_ARG, "ctr_rhopi_sigmapi_sets: null or misaligned pointer");
  for (int k = 0; k < 2 * nset; k++)
    if (sets[k] < 0 || sets[k] >= nphi)
      return ctr::fail(CTR_ERR_ARG, "ctr_rhopi_sigmapi_sets: elemental index %d not in [0,%d)", sets[k], nphi);
  return ctr::rhopi_sigmapi_core(nev, nt, tf_begin, tf_end, prop_rows, prop_diag, ctr::elems(nev, phi, nphi),
                                 mom5_p1p2, mom2_p1p2, nset, sets, {0, 1, 2}, rhopi, triangle, hor_fish,
                                 (cudaStream_t)stream, engine, true, nullptr, nullptr);
}

int ctr_loop_unity(int engine, int nev, int nt, const double* prop_diag, const double* mom, double* loop,
                   void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, 0, nt));
  if (!aligned(prop_diag) || !aligned(mom) || !aligned(loop)) return ctr::fail(CTR_ERR_ARG, "ctr_loop_unity: bad pointer");
  return ctr::loop_unity_fp64(nev, nt, prop_diag, mom, loop, (cudaStream_t)stream);
}

int ctr_sigmapi(int engine, int nev, int nt, int tf_begin, int tf_end, const double* prop_rows,
                const double* prop_diag, const double* mom_p1, const double* mom_p2, const double* mom2_p1p2,
                double* hor_fish, double* triangle, void* stream) {
  CTR_TRY(chain_args(engine, nev, nt, tf_begin, tf_end));
  if (!aligned(prop_diag) || !aligned(mom_p1) || !aligned(mom_p2) || (triangle && (!aligned(prop_rows) ||
      !aligned(mom2_p1p2) || !aligned(triangle))) || (hor_fish && !aligned(hor_fish)))
    return ctr::fail(CTR_ERR_ARG, "ctr_sigmapi: null or misaligned pointer");
  int32_t set[2];
  const std::vector<ctr::Elem> el = ctr::elems(nev, {mom_p1, mom_p2}, set);
  return ctr::rhopi_sigmapi_core(nev, nt, tf_begin, tf_end, prop_rows, prop_diag, el, nullptr, mom2_p1p2, 1, set, {},
                                 nullptr, triangle, hor_fish, (cudaStream_t)stream, engine, false, nullptr, nullptr);
}

}  // extern "C"
