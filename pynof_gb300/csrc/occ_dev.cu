// Occupation optimiser on the device: E(gamma), dE/dgamma and the whole
// conjugate-gradient minimisation over gamma at fixed J_MO, K_MO, H_core
// (occoptr, minimization.py:77-97, which calls scipy's CG on calcocce /
// calcoccg), without a host round trip per evaluation.
//
// One evaluation at a trial point gamma_t:
//  - occupations from the softmax parameterisation (ocupacion_softmax,
//    pnof.py:770-809; the strong occupation of pair i written at index i as
//    the reference does) and the per-orbital GNOF quantities of CJCKD8
//    (pnof.py:350-422): n, nd = n F(n_s), sqrt(nd), fi = sqrt(n (1 - n)) and
//    its derivative;
//  - the pair sums over (a, b) from different pairs (calce, pnof.py:905-929,
//    and the gradient of calcoccg, pnof.py:1004-1033 with der_CJCKD8,
//    pnof.py:425-525), a CTA per (32 orbitals a, 16 orbitals b) item, lanes over
//    a so that J[b][a] and K[b][a] are read coalesced.  The terms of a are
//    linear in five weighted sums over b (n_b J_ba, n_b K_ba, and over the
//    dynamic / static pairs fi_b K_ba, +-nd12_b K_ba, nd_b K_ba): at most five
//    FMAs per pair.  The last CTA to finish an a-group (an atomic count per
//    group, no waiting) adds the group's items; other CTAs take the same-pair
//    terms' roots and products meanwhile;
//  - the last CTA of all takes the step: the chain rule through nd = n F(n_s),
//    g = dn^T e, and the energy -- the assembly of the host loop of
//    occ_host.cu, summed in pairwise trees --, the minimiser's state, and the
//    next trial point's occupations.
//
// GB300 issues an FP64 warp instruction in 64 clocks per scheduler, whatever its
// lanes and its independent chains (an add or FMA one, a division or square root
// 10, exp 17), so the work is laid out for few FP64 warp instructions on any one
// scheduler: see occ_eval_kernel.
//
// The minimiser is scipy's CG as scipy 1.18 runs it: Polak-Ribiere+ with the
// sufficient-descent check, the first trial step from the previous decrease,
// and the line search of More & Thuente (ACM TOMS 20 (1994) 286-307; strong
// Wolfe with c1 = 1e-4, c2 = 0.4, xtol 1e-14, steps in [1e-100, 1e100], at most
// 100 calls), as a state machine that each evaluation advances by one
// step.  Where scipy would try its second line search (a failed search,
// or a step without sufficient descent), the state machine restarts from
// steepest descent once and otherwise stops at the current point.
//
// One CUDA graph per workspace runs a whole minimisation: an init kernel, a
// WHILE conditional node whose body is eight evaluations (the step clears the
// condition when the minimiser stops and the kernels after it return at once),
// then the occupations and C^J, C^K at the result.  The
// number of evaluations is capped at 1 + 200 (maxiter + 1): a minimiser that
// reaches the cap reports success -1.  The host-driven form
// (gb_occ_minimize_dev_sync) replays an ordinary graph of eight evaluations instead
// of the conditional node and reads the phase back after each replay.
//
// All arithmetic is FP64 (GB300's FP64 rate is low, so the O(nbf5^2) pair
// work is spread over the whole GPU and the single-CTA work is O(nbf5)).
// Closed shell without singly occupied orbitals (MSpin = 0, nsoc = 0).
#include <cmath>
#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

#include "gb_common.cuh"

namespace {

constexpr int kStepThreads = 256;  // one-CTA kernels; the sums of a step run over 256 threads
constexpr int kMinBlocks = 1;
constexpr int kEvalThreads = 384;  // evaluation kernel: ten warps of sums, two for the roots
constexpr int kUnroll = 8;         // evaluations per round of the WHILE node
constexpr int kCjckCtas = 2 * 152;
constexpr int kBch = 16;           // orbitals b per item of an evaluation
constexpr int kPairOrbs = 320;     // orbitals of a pair CTA whose roots it keeps in shared memory
constexpr size_t kStageSmem = 100 * 1024;  // a step's arrays are worked on in shared memory up to here
constexpr double kHCut = 0.02 * 1.4142135623730951;
// line search constants
constexpr double kFtol = 1e-4, kGtol = 0.4, kXtol = 1e-14, kStpMin = 1e-100, kStpMax = 1e100;
constexpr double kXtrapL = 1.1, kXtrapU = 4.0, kP5 = 0.5, kP66 = 0.66;
constexpr int kMaxCalls = 100;

enum { MODE_MIN = 0, MODE_EVAL = 1 };
enum { PH_INIT = 0, PH_LS = 1, PH_DONE = 2 };
enum { T_FG = 0, T_CONV = 1, T_FAIL = 2, T_STOP = 3 };

// A step's arrays, contiguous in this order (in the workspace, and in shared
// memory while the step works on them): what lives from step to step, then what
// the evaluation leaves for the step.  Arrays over the logits are in gamma's order.
struct OccStage {
  double *x, *g, *p, *xt, *nw;                      // nv
  double *n, *nd;                                   // P
  double *F, *dF, *ns;                              // ndoc
  double *es, *e, *en;                              // P: energy term, dE/dn, dE/dnd
  double *ej, *u, *v, *ew, *rw, *kws, *ksw;         // nv: same-pair terms
  double *gt;                                       // nv
};

__host__ __device__ __forceinline__ size_t stage_kept(int P, int nv, int ndoc) {
  return (size_t)5 * nv + (size_t)2 * P + (size_t)3 * ndoc;
}
__host__ __device__ __forceinline__ size_t stage_read(int P, int nv, int ndoc) {
  return stage_kept(P, nv, ndoc) + (size_t)3 * P + (size_t)7 * nv;
}
__host__ __device__ __forceinline__ size_t stage_size(int P, int nv, int ndoc) {
  return stage_read(P, nv, ndoc) + nv;
}
__host__ __device__ __forceinline__ OccStage stage_at(double* b, int P, int nv, int ndoc) {
  OccStage w;
  w.x = b; w.g = w.x + nv; w.p = w.g + nv; w.xt = w.p + nv; w.nw = w.xt + nv;
  w.n = w.nw + nv; w.nd = w.n + P;
  w.F = w.nd + P; w.dF = w.F + ndoc; w.ns = w.dF + ndoc;
  w.es = w.ns + ndoc; w.e = w.es + P; w.en = w.e + P;
  w.ej = w.en + P; w.u = w.ej + nv; w.v = w.u + nv; w.ew = w.v + nv; w.rw = w.ew + nv;
  w.kws = w.rw + nv; w.ksw = w.kws + nv; w.gt = w.ksw + nv;
  return w;
}

struct OccArgs {
  const double *J, *K, *H, *gamma0;
  double *gamma_out, *grad_out, *res, *n_out, *cj_out, *ck_out;
  // workspace arrays
  double* stage;                                // stage_size doubles
  double *fi, *nd12;                            // P, at the result (C^J, C^K)
  double *sq, *rsq;                             // P, pairs of more than kPairOrbs orbitals
  double *part;                                 // 5 sums of 32 orbitals per item
  int *pair_of, *cls;                           // P
  unsigned int* grp;                            // per a-group: items done; then the CTAs done
  int P, no1, ndoc, ncwo, nv, nbc, maxiter, mode;
  double gtol;
};

// More-Thuente line search
struct OccSearch {
  double stp, finit, ginit, gtest, width, width1, stx, fx, gx, sty, fy, gy, stmin, stmax;
  int brackt, stage, calls;
};

struct OccState {
  OccArgs a;
  // conjugate gradients (delta = g.g, d0 = g.p of the next line search)
  double f, f_prev, gnorm, delta, d0;
  int k, nev, maxev, phase, restarted;
  OccSearch ls;
};

__device__ __forceinline__ int weak_of(const OccArgs& a, int p, int j) {
  return a.no1 + a.ndoc + (a.ndoc - p - 1) + a.ndoc * j;
}
__device__ __forceinline__ int gam_of(const OccArgs& a, int p, int j) { return (a.ndoc - p - 1) + a.ndoc * j; }

// x >= y for y > 0, on the integer units (false for a NaN)
__device__ __forceinline__ bool at_least(double x, double y) {
  const long long b = __double_as_longlong(x);
  return b >= __double_as_longlong(y) && b <= 0x7ff0000000000000LL;
}

// The block's sums of v[0..3] over the first kStepThreads threads (fixed tree) and
// the largest m (bits of a non-negative double: a NaN's are the largest), given to
// every thread.  The four sums share their adds: lanes of one half go on with one
// sum, lanes of the other half with another (6 + 3 adds instead of 20 + 12).
__device__ void block_sums(double (&v)[4], unsigned long long& m, double* sh) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  unsigned long long* shm = reinterpret_cast<unsigned long long*>(sh + 32);
  if (w < kStepThreads / 32) {
    const bool h16 = l & 16, h8 = l & 8;
    // every add below pairs the same lanes as a shfl_down tree of one sum would
    const double a0 = __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[1], 16) + (h16 ? v[1] : v[0]);
    const double a1 = __shfl_xor_sync(0xffffffffu, h16 ? v[2] : v[3], 16) + (h16 ? v[3] : v[2]);
    double t = __shfl_xor_sync(0xffffffffu, h8 ? a0 : a1, 8) + (h8 ? a1 : a0);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t = __shfl_xor_sync(0xffffffffu, t, o) + t;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, m, o);
      m = y > m ? y : m;
    }
    // lanes 0, 16: sums 0, 1; lanes 8, 24: sums 2, 3
    if ((l & 7) == 0) sh[((l >> 4) + ((l >> 3) & 1) * 2) * 8 + w] = t;
    if (l == 0) shm[w] = m;
  }
  __syncthreads();
  if (w == 0) {
    double t = sh[l];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t = __shfl_xor_sync(0xffffffffu, t, o) + t;
    m = shm[l & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, m, o);
      m = y > m ? y : m;
    }
    __syncwarp();
    if ((l & 7) == 0) sh[l >> 3] = t;
    if (l == 0) shm[0] = m;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = sh[q];
  m = shm[0];
}

// Softmax weight j (-1: of the strong orbital) of a pair with logits x[nd q] past
// exp's range: shifted by the largest one.
__device__ __noinline__ double shifted_softmax(const double* x, int nd, int nc, int j) {
  double top = -INFINITY;
  for (int q = 0; q < nc; ++q) top = fmax(top, x[nd * q]);
  double den = exp(-top);
  for (int q = 0; q < nc; ++q) den += exp(x[nd * q] - top);
  return (j < 0 ? exp(-top) : exp(x[nd * j] - top)) / den;
}

// ---- the trial point's occupations and F (all threads of one CTA): a thread per
// logit, and the last threads a thread per pair for n_s
__device__ void prep_point(const OccArgs& a, const OccStage& w, const double* __restrict__ x) {
  const int tid = threadIdx.x, nd = a.ndoc, nc = a.ncwo, nv = a.nv, nvr = (nv + 31) / 32 * 32;
  // one exponential per logit, all at once (a pair with a logit past exp's
  // range is redone with its largest logit below; a NaN stays one)
  const int r0 = tid % nd;
  double* ex = w.ew;  // free between a step and the next evaluation
  for (int t = tid; t < nv; t += blockDim.x) ex[t] = exp(x[t]);
  __syncthreads();
  for (int t = tid; t < nvr + nd; t += blockDim.x) {
    const bool strong = t >= nvr;
    if (!strong && t >= nv) continue;
    const int r = strong ? t - nvr : t == tid ? r0 : t % nd, p = nd - 1 - r;  // logits r + nd j
    bool shift = false;
#pragma unroll 4
    for (int q = 0; q < nc; ++q) shift |= at_least(x[r + nd * q], 700.0);
    double val;
    if (shift) {
      // logits past exp's range: the same softmax shifted by the largest one
      val = shifted_softmax(x + r, nd, nc, strong ? -1 : t / nd);
    } else {
      double den = 1.0;
#pragma unroll 4
      for (int q = 0; q < nc; ++q) den += ex[r + nd * q];
      val = (strong ? 1.0 : ex[t]) / den;
    }
    if (strong) {
      w.ns[p] = val;
      w.n[p] = val;
    } else {
      w.nw[t] = val;
      w.n[a.no1 + nd + t] = val;
    }
  }
  __syncthreads();
  for (int p = tid; p < nd; p += blockDim.x) {
    const int s = a.no1 + p;
    const double coc = (1.0 - w.n[s]) / kHCut;
    const double F = exp(-coc * coc);
    w.F[p] = F;
    w.dF[p] = 2.0 * coc / kHCut;  // (1/F) dF/dn_s
  }
  __syncthreads();
  for (int t = tid; t < nvr + nd; t += blockDim.x) {
    const bool strong = t >= nvr;
    if (!strong && t >= nv) continue;
    const int r = strong ? t - nvr : t == tid ? r0 : t % nd, p = nd - 1 - r;
    const int i = strong ? a.no1 + p : a.no1 + nd + t;
    w.nd[i] = w.n[i] * w.F[p];
  }
  __syncthreads();
}

__device__ __forceinline__ double root_fi(double ni) { return sqrt(fmax(ni * (1.0 - ni), 0.0)); }

// ---- the parts of an evaluation, spread over the GPU

// Count n parts of a CTA as done; true in every thread of the CTA that completes
// `all`.  What other CTAs wrote before they counted is then read past L1 (__ldcg).
__device__ bool last_of(unsigned int* count, unsigned n, unsigned all, int& flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    flag = atomicAdd(count, n) + n == all;
    __threadfence();
  }
  __syncthreads();
  return flag;
}

// Item (ag, bc): per orbital a of group ag, five weighted sums over the orbitals b
// of block bc that are of other pairs:
// A1 = sum n_b J_ba, A2 = sum n_b K_ba and, over the pairs with the GNOF
// dynamic / static terms (a strong and b weak, or a weak and b not core),
// A3 = sum fi_b K_ba, A4 = sum s_ab nd12_b K_ba (s = -1 weak-weak),
// A5 = sum nd_b K_ba.  A warp per sum and parity of b.  The last item of a group
// adds the group's and forms the orbitals' energy and gradient terms, linear in
// the sums; true from it.
__device__ bool eval_item(const OccArgs& a, const OccStage& w, int ag, int bc, double (*red)[32], int& flag) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, P = a.P, nbc = a.nbc;
  const int i = ag * 32 + lane;
  const bool live = i < P;
  const int ii = live ? i : P - 1;
  const int b0 = bc * kBch;
  double(*sb)[32] = red + 10;  // [n, nd | fi, nd12][b]
  const double ni = w.n[ii], ndi = w.nd[ii];
  double(*ra)[32] = red + 12;  // for the group's last item: fi, fid, nd12, d of a
  if (warp == 10) {
    // the roots of the item's orbitals b: fi in the lower lanes, nd12 in the upper
    const int b = min(b0 + (lane & 15), P - 1);
    const double n = w.n[b], nd = w.nd[b];
    const double r = sqrt(lane < 16 ? fmax(n * (1.0 - n), 0.0) : nd);
    sb[1][lane] = r;
    if (lane < 16) {
      sb[0][lane] = n;
      sb[0][16 + lane] = nd;
    }
  }
  if (warp == 11) {
    const double fi = root_fi(ni);
    ra[0][lane] = fi;
    ra[1][lane] = ii < a.no1 ? 0.0 : (1.0 - 2.0 * ni) / (2.0 * fmax(fi, 1e-15));
    ra[2][lane] = sqrt(ndi);
    ra[3][lane] = 2.0 * a.H[ii] + a.J[(size_t)ii * P + ii];
  }
  const int k = warp >> 1, par = warp & 1;
  double m[kBch / 2];
  unsigned use = 0, neg = 0;
  if (warp < 10) {
    const double* M = k == 0 ? a.J : a.K;
    const int pa = a.pair_of[ii], ca = a.cls[ii];
#pragma unroll
    for (int u = 0; u < kBch / 2; ++u) {
      const int bb = b0 + 2 * u + par, b = min(bb, P - 1);
      m[u] = M[(size_t)b * P + ii];
      const int cb = a.cls[b];
      const bool ok = bb < P && b != ii && !(pa >= 0 && a.pair_of[b] == pa);
      const bool chi = ok && ((ca == 1 && cb == 2) || (ca == 2 && cb >= 1));
      if (k < 2 ? ok : chi) use |= 1u << u;
      if (k == 3 && ca == 2 && cb == 2) neg |= 1u << u;
    }
  }
  __syncthreads();
  if (warp < 10) {
    const double* wt = k < 2 ? sb[0] : k == 2 ? sb[1] : k == 3 ? sb[1] + 16 : sb[0] + 16;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < kBch / 2; ++u) {
      double wb = (use >> u) & 1 ? wt[2 * u + par] : 0.0;
      if ((neg >> u) & 1) wb = -wb;
      s = fma(wb, m[u], s);
    }
    red[warp][lane] = s;
  }
  __syncthreads();
  if (warp < 5)
    __stcg(a.part + ((size_t)(ag * nbc + bc) * 5 + warp) * 32 + lane, red[2 * warp][lane] + red[2 * warp + 1][lane]);
  if (!last_of(a.grp + ag, 1u, (unsigned)nbc, flag)) return false;
  // the last of the group's nbc items adds them up (the counter is left at zero
  // for the next evaluation)
  if (tid == 0) a.grp[ag] = 0;
  if (warp < 5) {
    const double* r = a.part + ((size_t)ag * nbc * 5 + warp) * 32 + lane;
    double t = 0.0;
    for (int c0 = 0; c0 < nbc; c0 += 16) {
      double y[16];
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (c0 + q < nbc) y[q] = __ldcg(r + (size_t)(c0 + q) * 160);
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (c0 + q < nbc) t += y[q];
    }
    red[warp][lane] = t;
  }
  __syncthreads();
  if (live) {
    const double A1 = red[0][lane], A2 = red[1][lane], A3 = red[2][lane], A4 = red[3][lane], A5 = red[4][lane];
    const double d = ra[3][lane];
    // pairs (i, b), b of another pair: sum_b 2 n_i n_b J_bi - C^K_ib K_bi
    if (warp == 0) w.es[i] = ni * d + (2.0 * ni * A1 - ni * A2 - ra[0][lane] * A3 - ra[2][lane] * A4 + ndi * A5);
    if (warp == 1) w.e[i] = d + 4.0 * A1 - 2.0 * A2 - 2.0 * ra[1][lane] * A3;
    if (warp == 2) w.en[i] = -2.0 * (A4 / (2.0 * fmax(ra[2][lane], 1e-15)) - A5);
  }
  return true;
}

// The terms inside pairs p0 <= p < p1 that do not wait for the sums.  C^J = 0;
// C^K = sqrt(n_s n_w) (strong-weak), -sqrt(n_w n_w') (weak-weak).
__device__ void eval_pairs(const OccArgs& a, const OccStage& w, int p0, int p1, double* root) {
  const int tid = threadIdx.x, nc = a.ncwo, np = p1 - p0, P = a.P;
  const bool near = np * (nc + 1) <= kPairOrbs;
  double *sq = near ? root : a.sq, *rsq = near ? root + kPairOrbs : a.rsq;
  // orbital q of the pairs: row q / np (0: strong, 1 + j: weak) of pair p0 + q % np
  const int base = near ? 0 : p0 * (nc + 1);
  for (int q = tid; q < np * (nc + 1); q += blockDim.x) {
    const int j = q / np, p = p0 + q - j * np;
    const double ni = w.n[j == 0 ? a.no1 + p : weak_of(a, p, j - 1)];
    const double r = sqrt(ni);
    sq[base + q] = r;
    rsq[base + q] = ni >= 1e-15 ? 1.0 / r : 1.0 / sqrt(1e-15);
  }
  __syncthreads();
  for (int q = tid; q < np * nc; q += blockDim.x) {
    const int j = q / np, pl = q - j * np, p = p0 + pl;
    const int s = a.no1 + p, o = weak_of(a, p, j), t = gam_of(a, p, j);
    const double Kws = a.K[(size_t)o * P + s], Ksw = a.K[(size_t)s * P + o];
    const double sqs = sq[base + pl], rs = rsq[base + pl];
    const double sqw = sq[base + (j + 1) * np + pl], rw = rsq[base + (j + 1) * np + pl];
    double ew = 0.0, ej = -(sqs * sqw) * (Kws + Ksw);
#pragma unroll 4
    for (int j2 = 0; j2 < nc; ++j2) {
      if (j2 == j) continue;
      const double Kw2w = a.K[(size_t)weak_of(a, p, j2) * P + o];
      const double s2 = sq[base + (j2 + 1) * np + pl];
      ej += sqw * s2 * Kw2w;
      ew += s2 * Kw2w;
    }
    w.ej[t] = ej;
    w.u[t] = sqw * rs;
    w.v[t] = sqs * rw;
    w.ew[t] = ew;
    w.rw[t] = rw;
    w.kws[t] = Kws;
    w.ksw[t] = Ksw;
  }
}

// (weak orbital j of pair p = nd - 1 - r is no1 + nd + r + nd j, its logit r + nd j)
// ---- gradient at the trial point from the evaluation's parts (one CTA); E's share
// of each thread.  A thread per logit, the threads past kStepThreads a pair each.
__device__ double assemble(const OccArgs& a, const OccStage& w) {
  const int tid = threadIdx.x, nd = a.ndoc, nv = a.nv, nc = a.ncwo;
  const int pt = tid - kStepThreads, pn = kEvalThreads - kStepThreads, j0 = tid / nd;
  // the same-pair terms, then the chain dE/dnd to the occupations (nd_s = n_s
  // F(n_s), nd_w = n_w F(n_s)); u: the weak orbitals' share of the strong one
  for (int p = pt; p >= 0 && p < nd; p += pn) {
    const int s = a.no1 + p;
    double e_s = w.e[s];
#pragma unroll 4
    for (int j = 0; j < nc; ++j) {
      const int t = nd - p - 1 + nd * j;
      e_s -= w.u[t] * w.kws[t];
    }
    const double F = w.F[p], dF = w.dF[p];
    w.e[s] = e_s + w.en[s] * F * (1.0 + w.n[s] * dF);
  }
  if (tid < kStepThreads)
    for (int t = tid; t < nv; t += kStepThreads) {
      const int j = t == tid ? j0 : t / nd, r = t - j * nd, p = nd - 1 - r, o = a.no1 + nd + t;
      const double F = w.F[p], en = w.en[o];
      double e = w.e[o] - w.v[t] * w.ksw[t] + w.rw[t] * w.ew[t];
      w.e[o] = e + en * F;
      w.rw[t] = en * w.n[o] * F;
    }
  __syncthreads();
  for (int p = pt; p >= 0 && p < nd; p += pn) {
    const int s = a.no1 + p;
    const double dF = w.dF[p];
    double e_s = w.e[s];
#pragma unroll 4
    for (int j = 0; j < nc; ++j) e_s += w.rw[nd - p - 1 + nd * j] * dF;
    w.e[s] = e_s;
  }
  double es = 0.0;
  if (tid < kStepThreads) {
    for (int i = tid; i < a.P; i += kStepThreads) es += w.es[i];
    for (int p = tid; p < nd; p += kStepThreads) {
      double ep = 0.0;
#pragma unroll 4
      for (int j = 0; j < nc; ++j) ep += w.ej[nd - p - 1 + nd * j];
      es += ep;
    }
  }
  __syncthreads();
  // g = dn^T e (row p of dn holds the strong occupation)
  if (tid < kStepThreads)
    for (int t = tid; t < nv; t += kStepThreads) {
      const int j = t == tid ? j0 : t / nd, r = t - j * nd, p = nd - 1 - r;
      const int weak = a.no1 + nd + r;  // its pair's weak orbitals: + nd j
      double wsum = 0.0;
#pragma unroll 4
      for (int q = 0; q < nc; ++q) wsum += w.nw[r + nd * q] * w.e[weak + nd * q];
      const double o = w.nw[t];
      w.gt[t] = -w.ns[p] * o * w.e[p] + o * w.e[weak + nd * j] - o * wsum;
    }
  return es;
}

// ---- More & Thuente, one safeguarded step (section 4 of the paper), by all lanes
// of a warp with the same values: a warp instruction costs the same for one lane as
// for 32, so independent divisions are lanes of one (10 warp instructions each)

// num0 / den0 and num1 / den1
__device__ __forceinline__ void quotients(double num0, double den0, double num1, double den1, double& q0, double& q1) {
  const bool odd = threadIdx.x & 1;
  const double q = (odd ? num1 : num0) / (odd ? den1 : den0);
  q0 = __shfl_sync(0xffffffffu, q, 0);
  q1 = __shfl_sync(0xffffffffu, q, 1);
}

// (theta / s)^2 - (d1 / s) (d2 / s)
__device__ __forceinline__ double discriminant(double theta, double d1, double d2, double s) {
  const int l = threadIdx.x & 31;
  const double q = (l == 0 ? theta : l == 1 ? d1 : d2) / s;
  const double t = __shfl_sync(0xffffffffu, q, 0), a = __shfl_sync(0xffffffffu, q, 1),
               b = __shfl_sync(0xffffffffu, q, 2);
  return fma(-a, b, __dmul_rn(t, t));  // (the rounding that the search has always had)
}

// d / |d|: +-1, or a NaN where d is zero or not finite
__device__ __forceinline__ double unit_sign(double d) {
  const long long b = __double_as_longlong(d), m = b & 0x7fffffffffffffffLL;
  return m == 0 || m >= 0x7ff0000000000000LL ? NAN : copysign(1.0, d);
}

__device__ void dcstep(double& stx, double& fx, double& dx, double& sty, double& fy, double& dy, double& stp,
                       double fp, double dp, int& brackt, double stpmin, double stpmax) {
  const double sgnd = dp * unit_sign(dx);
  double stpf;
  if (fp > fx) {
    double third, slope;
    quotients(3.0 * (fx - fp), stp - stx, fx - fp, stp - stx, third, slope);
    const double theta = third + dx + dp;
    const double s = fmax(fmax(fabs(theta), fabs(dx)), fabs(dp));
    double gamma = s * sqrt(discriminant(theta, dx, dp, s));
    if (stp < stx) gamma = -gamma;
    const double p = (gamma - dx) + theta;
    const double q = ((gamma - dx) + gamma) + dp;
    double r, rq;
    quotients(p, q, dx, slope + dx, r, rq);
    const double stpc = stx + r * (stp - stx);
    const double stpq = stx + (rq / 2.0) * (stp - stx);
    stpf = fabs(stpc - stx) < fabs(stpq - stx) ? stpc : stpc + (stpq - stpc) / 2.0;
    brackt = 1;
  } else if (sgnd < 0.0) {
    const double theta = 3.0 * (fx - fp) / (stp - stx) + dx + dp;
    const double s = fmax(fmax(fabs(theta), fabs(dx)), fabs(dp));
    double gamma = s * sqrt(discriminant(theta, dx, dp, s));
    if (stp > stx) gamma = -gamma;
    const double p = (gamma - dp) + theta;
    const double q = ((gamma - dp) + gamma) + dx;
    double r, rq;
    quotients(p, q, dp, dp - dx, r, rq);
    const double stpc = stp + r * (stx - stp);
    const double stpq = stp + rq * (stx - stp);
    stpf = fabs(stpc - stp) > fabs(stpq - stp) ? stpc : stpq;
    brackt = 1;
  } else if (fabs(dp) < fabs(dx)) {
    const double theta = 3.0 * (fx - fp) / (stp - stx) + dx + dp;
    const double s = fmax(fmax(fabs(theta), fabs(dx)), fabs(dp));
    const double disc = discriminant(theta, dx, dp, s);
    double gamma = s * sqrt(disc > 0.0 ? disc : 0.0);
    if (stp > stx) gamma = -gamma;
    const double p = (gamma - dp) + theta;
    const double q = (gamma + (dx - dp)) + gamma;
    double r, rq;
    quotients(p, q, dp, dp - dx, r, rq);
    double stpc;
    if (r < 0.0 && gamma != 0.0)
      stpc = stp + r * (stx - stp);
    else if (stp > stx)
      stpc = stpmax;
    else
      stpc = stpmin;
    const double stpq = stp + rq * (stx - stp);
    if (brackt) {
      stpf = fabs(stpc - stp) < fabs(stpq - stp) ? stpc : stpq;
      if (stp > stx)
        stpf = fmin(stp + kP66 * (sty - stp), stpf);
      else
        stpf = fmax(stp + kP66 * (sty - stp), stpf);
    } else {
      stpf = fabs(stpc - stp) > fabs(stpq - stp) ? stpc : stpq;
      stpf = fmin(stpmax, stpf);
      stpf = fmax(stpmin, stpf);
    }
  } else {
    if (brackt) {
      const double theta = 3.0 * (fp - fy) / (sty - stp) + dy + dp;
      const double s = fmax(fmax(fabs(theta), fabs(dy)), fabs(dp));
      double gamma = s * sqrt(discriminant(theta, dy, dp, s));
      if (stp > sty) gamma = -gamma;
      const double p = (gamma - dp) + theta;
      const double q = ((gamma - dp) + gamma) + dy;
      const double r = p / q;
      stpf = stp + r * (sty - stp);
    } else if (stp > stx) {
      stpf = stpmax;
    } else {
      stpf = stpmin;
    }
  }
  if (fp > fx) {
    sty = stp;
    fy = fp;
    dy = dp;
  } else {
    if (sgnd < 0.0) {
      sty = stx;
      fy = fx;
      dy = dx;
    }
    stx = stp;
    fx = fp;
    dx = dp;
  }
  stp = stpf;
}

__device__ int ls_fg(OccSearch& S, double stp) {
  if (!isfinite(stp) || S.calls >= kMaxCalls) return T_FAIL;
  S.stp = stp;
  return T_FG;
}

__device__ int ls_start(OccSearch& S, double stp, double f, double g) {
  S.calls = 1;
  if (stp < kStpMin || stp > kStpMax || g >= 0.0) return T_FAIL;
  S.brackt = 0;
  S.stage = 1;
  S.finit = f;
  S.ginit = g;
  S.gtest = kFtol * g;
  S.width = kStpMax - kStpMin;
  S.width1 = S.width / kP5;
  S.stx = 0.0;
  S.fx = f;
  S.gx = g;
  S.sty = 0.0;
  S.fy = f;
  S.gy = g;
  S.stmin = 0.0;
  S.stmax = stp + kXtrapU * stp;
  return ls_fg(S, stp);
}

__device__ int ls_step(OccSearch& S, double f, double g) {
  S.calls += 1;
  double stp = S.stp;
  const double ftest = S.finit + stp * S.gtest;
  if (S.stage == 1 && f <= ftest && g >= 0.0) S.stage = 2;
  const bool warn = (S.brackt && (stp <= S.stmin || stp >= S.stmax)) ||
                    (S.brackt && S.stmax - S.stmin <= kXtol * S.stmax) ||
                    (stp == kStpMax && f <= ftest && g <= S.gtest) ||
                    (stp == kStpMin && (f > ftest || g >= S.gtest));
  if (f <= ftest && fabs(g) <= kGtol * (-S.ginit)) return T_CONV;
  if (warn) return T_FAIL;
  if (S.stage == 1 && f <= S.fx && f > ftest) {
    // the modified function psi(a) = phi(a) - phi(0) - ftol phi'(0) a
    double fxm = S.fx - S.stx * S.gtest, fym = S.fy - S.sty * S.gtest;
    double gxm = S.gx - S.gtest, gym = S.gy - S.gtest;
    dcstep(S.stx, fxm, gxm, S.sty, fym, gym, stp, f - stp * S.gtest, g - S.gtest, S.brackt, S.stmin, S.stmax);
    S.fx = fxm + S.stx * S.gtest;
    S.fy = fym + S.sty * S.gtest;
    S.gx = gxm + S.gtest;
    S.gy = gym + S.gtest;
  } else {
    dcstep(S.stx, S.fx, S.gx, S.sty, S.fy, S.gy, stp, f, g, S.brackt, S.stmin, S.stmax);
  }
  if (S.brackt) {
    if (fabs(S.sty - S.stx) >= kP66 * S.width1) stp = S.stx + kP5 * (S.sty - S.stx);
    S.width1 = S.width;
    S.width = fabs(S.sty - S.stx);
    S.stmin = fmin(S.stx, S.sty);
    S.stmax = fmax(S.stx, S.sty);
  } else {
    S.stmin = stp + kXtrapL * (stp - S.stx);
    S.stmax = stp + kXtrapU * (stp - S.stx);
  }
  stp = fmin(fmax(stp, kStpMin), kStpMax);
  if ((S.brackt && (stp <= S.stmin || stp >= S.stmax)) || (S.brackt && S.stmax - S.stmin <= kXtol * S.stmax))
    stp = S.stx;
  return ls_fg(S, stp);
}

// a search's first trial step, from the previous decrease
__device__ __forceinline__ double first_step(double f, double f_prev, double d0) {
  double alpha1 = 1.0;
  if (d0 != 0.0) {
    const double v = 1.01 * 2 * (f - f_prev) / d0;
    alpha1 = v < 1.0 ? v : 1.0;  // min(1, v) with Python's argument order
    if (alpha1 < 0.0) alpha1 = 1.0;
  }
  return alpha1;
}

// ---- kernels
__global__ void __launch_bounds__(kStepThreads, kMinBlocks) occ_init_kernel(OccState* st, OccArgs args) {
  OccState& S = *st;
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.a = args;
    S.phase = PH_INIT;
    S.nev = 0;
    S.k = 0;
    S.restarted = 0;
    S.maxev = 1 + 200 * (args.maxiter + 1);
  }
  const OccArgs& a = args;
  const OccStage w = stage_at(a.stage, a.P, a.nv, a.ndoc);
  const int nb = a.no1 + a.ndoc;
  for (int i = tid; i < a.P; i += kStepThreads) {
    w.n[i] = 0.0;
    w.nd[i] = 0.0;
    a.pair_of[i] = -1;
    a.cls[i] = i < a.no1 ? 0 : (i < nb ? 1 : 2);  // 1: strong set S, 2: weak set W
  }
  __syncthreads();
  for (int g = tid; g < (a.P + 31) / 32 + 1; g += kStepThreads) a.grp[g] = 0u;
  for (int p = tid; p < a.ndoc; p += kStepThreads) {
    a.pair_of[a.no1 + p] = p;
    for (int j = 0; j < a.ncwo; ++j) a.pair_of[weak_of(a, p, j)] = p;
  }
  for (int i = tid; i < a.nv; i += kStepThreads) {
    w.x[i] = a.gamma0[i];
    w.xt[i] = a.gamma0[i];
  }
  __syncthreads();
  prep_point(a, w, w.xt);
}

__device__ void finish(OccState& S, const OccStage& w, double success, cudaGraphConditionalHandle h, int cond) {
  const OccArgs& a = S.a;
  for (int i = threadIdx.x; i < a.nv; i += blockDim.x) a.gamma_out[i] = w.x[i];
  if (threadIdx.x == 0) {
    a.res[0] = S.f;
    a.res[1] = S.k;
    a.res[2] = S.nev;
    a.res[3] = success;
    a.res[4] = S.gnorm;
    S.phase = PH_DONE;
    if (cond) cudaGraphSetConditional(h, 0);
  }
}

__device__ void step_body(OccState& S, const OccStage& w, double* sh, int& s_act, cudaGraphConditionalHandle h,
                          int cond);

// CTAs of an evaluation: an item per (a-group, b-block), then the pair CTAs
__host__ __device__ __forceinline__ int pairs_per_cta(int ncwo) { return ncwo + 1 < 128 ? 128 / (ncwo + 1) : 1; }

// One evaluation and the step it leads to.  The CTAs spread the sums and roots over
// the GPU; the last of them to finish (counts, no waiting) takes the step.  What
// bounds it is the FP64 issue rate: 64 clocks per warp instruction and scheduler
// whatever the lanes or the independent chains in it, so each scheduler is given as
// few as possible (a warp per sum and parity: 8 FMAs instead of 80; a thread per
// logit instead of per pair; four block sums in one tree; maxima and range tests on
// the integer units) and the step's arrays are kept in shared memory.  As a kernel
// of one-warp items followed by a kernel of one CTA, an evaluation of 150 orbitals
// took 43 us (14 us and 26 us, and the launches), now 22 us: 8 us for the parts, each
// exchange between CTAs (a fence, a count, loads past L1) 1 to 2 us of them, 9 us for the
// step (exponentials, divisions and the line search follow one another), 1.3 us between
// launches.
__global__ void __launch_bounds__(kEvalThreads, kMinBlocks)
    occ_eval_kernel(OccState* st, cudaGraphConditionalHandle h, int cond, int staged) {
  extern __shared__ double stage_sh[];
  __shared__ double red[16][32];
  __shared__ double root[2 * kPairOrbs];
  __shared__ double sh[40];
  __shared__ int s_act;
  // the step works on a copy in shared memory: its scalars and the array
  // pointers are read there, not from global memory behind every store
  __shared__ OccState S;
  const int tid = threadIdx.x;
  const OccArgs g = st->a;
  if (st->phase == PH_DONE) {
    if (blockIdx.x == 0 && tid == 0 && cond) cudaGraphSetConditional(h, 0);
    return;
  }
  const int P = g.P, nv = g.nv, ndoc = g.ndoc, nag = (P + 31) / 32, items = nag * g.nbc;
  double* stage = g.stage;
  const OccStage wg = stage_at(stage, P, nv, ndoc);
  const int ppc = pairs_per_cta(g.ncwo), npc = (ndoc + ppc - 1) / ppc;
  bool mine = false;  // this CTA finished a group or a block of pairs
  int parts = 0;
  for (int it = blockIdx.x; it < items + npc; it += gridDim.x) {
    if (it < items) {
      const int ag = it / g.nbc;
      mine = eval_item(g, wg, ag, it - ag * g.nbc, red, s_act);
    } else {
      const int p0 = (it - items) * ppc;
      eval_pairs(g, wg, p0, min(ndoc, p0 + ppc), root);
      mine = true;
    }
    parts += mine;
    __syncthreads();
  }
  if (parts == 0) return;
  // the state and the arrays kept from the last step do not wait for the other
  // CTAs: their loads are under way while the parts are counted
  constexpr int kAhead = 4;
  const int kept = (int)stage_kept(P, nv, ndoc);
  const unsigned long long* sw = reinterpret_cast<const unsigned long long*>(st);
  static_assert(sizeof(OccState) / 8 <= kEvalThreads && sizeof(OccState) % 8 == 0, "a thread per word of the state");
  const bool has_word = tid < (int)(sizeof(OccState) / 8);
  const unsigned long long word = has_word ? sw[tid] : 0;
  double ahead[kAhead];
#pragma unroll
  for (int q = 0; q < kAhead; ++q) {
    const int i = tid + q * kEvalThreads;
    ahead[q] = staged && i < kept ? stage[i] : 0.0;
  }
  if (!last_of(g.grp + nag, (unsigned)parts, (unsigned)(nag + npc), s_act)) return;
  if (has_word) reinterpret_cast<unsigned long long*>(&S)[tid] = word;
  if (tid == 0) g.grp[nag] = 0;
  if (staged) {
    const int total = (int)stage_read(P, nv, ndoc);
#pragma unroll 4
    for (int i = kept + tid; i < total; i += kEvalThreads) stage_sh[i] = __ldcg(stage + i);
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      const int i = tid + q * kEvalThreads;
      if (i < kept) stage_sh[i] = ahead[q];
    }
    for (int i = tid + kAhead * kEvalThreads; i < kept; i += kEvalThreads) stage_sh[i] = stage[i];
  }
  __syncthreads();
  step_body(S, staged ? stage_at(stage_sh, P, nv, ndoc) : wg, sh, s_act, h, cond);
  __syncthreads();
  if (has_word) reinterpret_cast<unsigned long long*>(st)[tid] = reinterpret_cast<unsigned long long*>(&S)[tid];
  if (staged)
    for (int i = tid; i < kept; i += kEvalThreads) stage[i] = stage_sh[i];
}

__device__ void step_body(OccState& S, const OccStage& w, double* sh, int& s_act, cudaGraphConditionalHandle h,
                          int cond) {
  const OccArgs& a = S.a;
  const int tid = threadIdx.x;
  // g1.p (the search's slope), (g1 - g).g1, g1.g1 at the trial point, E and max |g1|
  // in one reduction
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  unsigned long long top = 0;
  v[3] = assemble(a, w);
  if (tid < kStepThreads) {
    const bool searching = S.phase == PH_LS;
    for (int i = tid; i < a.nv; i += kStepThreads) {
      const double gi = w.gt[i];
      if (searching) {
        v[0] += gi * w.p[i];
        v[1] += (gi - w.g[i]) * gi;
      }
      v[2] += gi * gi;
      const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(gi));
      top = b > top ? b : top;
    }
  }
  block_sums(v, top, sh);
  const double E = v[3], gmax = __longlong_as_double((long long)top);
  if (tid == 0) S.nev += 1;
  if (a.mode == MODE_EVAL) {
    for (int i = tid; i < a.nv; i += blockDim.x) {
      if (a.grad_out) a.grad_out[i] = w.gt[i];
      w.x[i] = w.xt[i];
    }
    if (tid == 0) {
      S.f = E;
      S.gnorm = gmax;
    }
    __syncthreads();
    finish(S, w, 1.0, h, cond);
    return;
  }
  enum { A_BEGIN, A_FAIL, A_EVAL, A_STOP_OK, A_STOP_FAIL, A_STOP_CAP };
  int act;
  bool known = false;  // the next search's first step is in sh[39]
  if (S.phase == PH_INIT) {
    for (int i = tid; i < a.nv; i += blockDim.x) {
      const double gi = w.gt[i];
      w.g[i] = gi;
      w.p[i] = -gi;
    }
    if (tid == 0) {
      S.f = E;
      S.f_prev = E + sqrt(v[2]) / 2.0;
      S.gnorm = gmax;
      S.delta = v[2];
      S.d0 = -v[2];
    }
    __syncthreads();  // every thread reads S.gnorm next
    act = A_BEGIN;
  } else {
    // the search's step, and on another scheduler what an accepted point leads to
    if (tid < 32) {
      OccSearch ls = S.ls;
      const int task = ls_step(ls, E, v[0]);
      __syncwarp();
      if (tid == 0) {
        S.ls = ls;
        s_act = task;
      }
    } else if (tid == 32) {
      const double r = v[1] / S.delta;
      const double beta = r > 0.0 ? r : 0.0;
      // p1 = -g1 + beta p: p1.g1 = -g1.g1 + beta g1.p
      const double pg = -v[2] + beta * v[0];
      sh[36] = beta;
      sh[37] = pg;
      sh[38] = gmax <= a.gtol || pg <= -0.01 * v[2] ? 1.0 : 0.0;
      sh[39] = first_step(E, S.f, pg);
    }
    __syncthreads();
    const int task = s_act;
    if (task == T_FG) {
      act = A_EVAL;
    } else if (task == T_CONV) {
      if (__double_as_longlong(sh[38]) != 0) {
        const double beta = sh[36];
        for (int i = tid; i < a.nv; i += blockDim.x) {
          const double gi = w.gt[i];
          w.x[i] = w.xt[i];
          w.p[i] = -gi + beta * w.p[i];
          w.g[i] = gi;
        }
        if (tid == 0) {
          S.f_prev = S.f;
          S.f = E;
          S.gnorm = gmax;
          S.delta = v[2];
          S.d0 = sh[37];
          S.k += 1;
          S.restarted = 0;
        }
        act = A_BEGIN;
        known = true;
      } else {
        act = A_FAIL;
      }
    } else {
      act = A_FAIL;
    }
    __syncthreads();
  }
  // at most: fail -> begin (restarted) -> fail -> stop
  for (int guard = 0; guard < 4; ++guard) {
    if (act == A_FAIL) {
      int ne = 0;
      for (int i = tid; i < a.nv; i += blockDim.x) ne |= (w.p[i] != -w.g[i]);
      const int alleq = __syncthreads_or(ne) == 0;
      if (S.restarted || alleq) {
        act = A_STOP_FAIL;
      } else {
        for (int i = tid; i < a.nv; i += blockDim.x) w.p[i] = -w.g[i];
        __syncthreads();
        if (tid == 0) {
          S.restarted = 1;
          S.d0 = -S.delta;  // p = -g
        }
        act = A_BEGIN;
      }
      __syncthreads();
    }
    if (act == A_BEGIN) {
      if (tid == 0) {
        if (!(S.gnorm > a.gtol) || S.k >= a.maxiter)
          s_act = T_STOP;
        else
          s_act = ls_start(S.ls, known ? sh[39] : first_step(S.f, S.f_prev, S.d0), S.f, S.d0);
      }
      known = false;
      __syncthreads();
      act = s_act == T_STOP ? A_STOP_OK : s_act == T_FG ? A_EVAL : A_FAIL;
      __syncthreads();
    }
    if (act != A_FAIL && act != A_BEGIN) break;
  }
  if (act == A_EVAL && S.nev >= S.maxev) act = A_STOP_CAP;
  if (act == A_EVAL) {
    const double stp = S.ls.stp;
    for (int i = tid; i < a.nv; i += blockDim.x) w.xt[i] = w.x[i] + stp * w.p[i];
    __syncthreads();
    prep_point(a, w, w.xt);
    if (tid == 0) S.phase = PH_LS;
    return;
  }
  __syncthreads();
  const double success = act == A_STOP_CAP ? -1.0 : (act == A_STOP_OK && S.gnorm <= a.gtol ? 1.0 : 0.0);
  finish(S, w, success, h, cond);
}

// the occupations at the result (one CTA), then C^J, C^K (grid)
__global__ void __launch_bounds__(kStepThreads, kMinBlocks) occ_final_kernel(const OccState* __restrict__ st) {
  const OccArgs& a = st->a;
  if (!a.n_out && !a.cj_out) return;
  const OccStage w = stage_at(a.stage, a.P, a.nv, a.ndoc);
  prep_point(a, w, w.x);
  for (int i = threadIdx.x; i < a.P; i += kStepThreads) {
    if (a.n_out) a.n_out[i] = w.n[i];
    a.fi[i] = root_fi(w.n[i]);
    a.nd12[i] = sqrt(w.nd[i]);
  }
}

// CJCKD8 (pnof.py:350-422) at the result's occupations, diagonals included:
// C^J = 2 n n^T, C^K = n n^T, plus on S x W, W x S, W x W the fi fi^T and
// +-nd12 nd12^T - nd nd^T terms; inside each pair block C^J = 0 and
// C^K = sqrt(n_s n_w) (strong-weak), -sqrt(n_w n_w') (weak-weak).  The
// elementwise order of the numpy expressions, without contraction.
__global__ void __launch_bounds__(kStepThreads, kMinBlocks) occ_cjck_kernel(const OccState* __restrict__ st) {
  const OccArgs& a = st->a;
  if (!a.cj_out || !a.ck_out) return;
  const int P = a.P, nb = a.no1 + a.ndoc, na = nb;
  const OccStage w = stage_at(a.stage, P, a.nv, a.ndoc);
  const long long total = (long long)P * P;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / P), j = (int)(t - (long long)i * P);
    const double ni = w.n[i], nj = w.n[j];
    double cj = __dmul_rn(2.0, __dmul_rn(ni, nj));
    double ck = __dmul_rn(ni, nj);
    const bool Si = i >= a.no1 && i < nb, Sj = j >= a.no1 && j < nb, Wi = i >= na, Wj = j >= na;
    if ((Si && Wj) || (Wi && Sj) || (Wi && Wj)) ck = __dadd_rn(ck, __dmul_rn(a.fi[i], a.fi[j]));
    if ((Si && Wj) || (Wi && Sj))
      ck = __dadd_rn(ck, __dsub_rn(__dmul_rn(a.nd12[i], a.nd12[j]), __dmul_rn(w.nd[i], w.nd[j])));
    if (Wi && Wj) ck = __dadd_rn(ck, __dsub_rn(-__dmul_rn(a.nd12[i], a.nd12[j]), __dmul_rn(w.nd[i], w.nd[j])));
    const int pi = a.pair_of[i], pj = a.pair_of[j];
    if (pi >= 0 && pi == pj) {
      const bool si = i == a.no1 + pi, sj = j == a.no1 + pj;
      if (!(si && sj)) {
        cj = 0.0;
        if (si || sj)
          ck = sqrt(__dmul_rn(w.n[si ? i : j], w.n[si ? j : i]));
        else
          ck = -sqrt(__dmul_rn(ni, nj));
      }
    }
    a.cj_out[t] = cj;
    a.ck_out[t] = ck;
  }
}

// ---- workspace and graphs
template <class Cv>
void occ_layout(Cv& c, int P, int ndoc, int ncwo, OccState** state, OccArgs& a) {
  const int nv = ndoc * ncwo, nbc = (P + kBch - 1) / kBch;
  *state = c.template take<OccState>(1);
  a.stage = c.template take<double>(stage_size(P, nv, ndoc));
  a.fi = c.template take<double>(P);
  a.nd12 = c.template take<double>(P);
  a.sq = c.template take<double>(P);
  a.rsq = c.template take<double>(P);
  a.part = c.template take<double>((size_t)5 * 32 * ((P + 31) / 32) * nbc);
  a.pair_of = c.template take<int>(P);
  a.cls = c.template take<int>(P);
  a.grp = c.template take<unsigned int>((P + 31) / 32 + 1);
  a.nv = nv;
  a.nbc = nbc;
}

struct OccGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaGraphNode_t init = nullptr;
  // host-driven form: kChunk evaluations as an ordinary graph
  cudaGraph_t chunk_graph = nullptr;
  cudaGraphExec_t chunk_exec = nullptr;
};

constexpr int kChunk = 8;  // evaluations per replay of the host-driven form

std::mutex g_mu;
// (context id, workspace, nbf5) -> graph; a context re-created after
// cudaDeviceReset has a new id, so a stale graph is never reused
std::map<std::tuple<unsigned long long, const void*, int>, OccGraph> g_graphs;

// One evaluation: a CTA per item and enough for the pairs of any structure of P
// orbitals (the kernel strides over what is left), with a step's arrays in shared
// memory where the largest such structure's fit.
cudaError_t add_eval_node(cudaGraphNode_t* node, cudaGraph_t g, cudaGraphNode_t prev, OccState* st, int P,
                          cudaGraphConditionalHandle h, int cond) {
  // nv <= P - ndoc: 13 nv + 5 P + 3 ndoc <= 18 P
  const size_t smem = (size_t)18 * P * sizeof(double);
  int staged = smem <= kStageSmem;
  cudaError_t e = cudaFuncSetAttribute((const void*)occ_eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kStageSmem);
  if (e != cudaSuccess) return e;
  const long long ctas = (long long)((P + 31) / 32) * ((P + kBch - 1) / kBch) + (P + 63) / 64 + 1;
  void* params[] = {&st, &h, &cond, &staged};
  cudaKernelNodeParams kp{};
  kp.func = (void*)occ_eval_kernel;
  kp.gridDim = dim3((unsigned)(ctas < 65535 ? ctas : 65535));
  kp.blockDim = dim3(kEvalThreads);
  kp.sharedMemBytes = staged ? (unsigned)smem : 0;
  kp.kernelParams = params;
  return cudaGraphAddKernelNode(node, g, prev ? &prev : nullptr, prev ? 1 : 0, &kp);
}

int build_graph(OccState* st, int P, OccGraph& og) {
  cudaGraph_t g = nullptr;
  GB_TRY(gb::cuda_status(cudaGraphCreate(&g, 0), "occ graph create"));
  auto fail = [&](cudaError_t e, const char* where) {
    cudaGraphDestroy(g);
    return gb::cuda_status(e, where);
  };
  OccArgs dummy{};
  void* ip[] = {&st, &dummy};
  cudaKernelNodeParams kp{};
  kp.func = (void*)occ_init_kernel;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(kStepThreads);
  kp.kernelParams = ip;
  cudaGraphNode_t init = nullptr, wn = nullptr, n4 = nullptr, n5 = nullptr;
  cudaError_t e = cudaGraphAddKernelNode(&init, g, nullptr, 0, &kp);
  if (e != cudaSuccess) return fail(e, "occ graph: init node");
  cudaGraphConditionalHandle h;
  e = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
  if (e != cudaSuccess) return fail(e, "occ graph: conditional handle");
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  e = cudaGraphAddNode(&wn, g, &init, nullptr, 1, &cp);
  if (e != cudaSuccess) return fail(e, "occ graph: while node");
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  void* sp[] = {&st};
  cudaGraphNode_t prev = nullptr;
  for (int u = 0; u < kUnroll; ++u) {
    cudaGraphNode_t n1 = nullptr;
    e = add_eval_node(&n1, body, prev, st, P, h, 1);
    if (e != cudaSuccess) return fail(e, "occ graph: evaluation node");
    prev = n1;
  }
  cudaKernelNodeParams fk{};
  fk.func = (void*)occ_final_kernel;
  fk.gridDim = dim3(1);
  fk.blockDim = dim3(kStepThreads);
  fk.kernelParams = sp;
  e = cudaGraphAddKernelNode(&n4, g, &wn, 1, &fk);
  if (e != cudaSuccess) return fail(e, "occ graph: final node");
  cudaKernelNodeParams ck{};
  ck.func = (void*)occ_cjck_kernel;
  ck.gridDim = dim3(kCjckCtas);
  ck.blockDim = dim3(kStepThreads);
  ck.kernelParams = sp;
  e = cudaGraphAddKernelNode(&n5, g, &n4, 1, &ck);
  if (e != cudaSuccess) return fail(e, "occ graph: cjck node");
  cudaGraphExec_t exec = nullptr;
  e = cudaGraphInstantiate(&exec, g, 0);
  if (e != cudaSuccess) return fail(e, "occ graph: instantiate");
  og.graph = g;
  og.exec = exec;
  og.init = init;
  return GB_OK;
}

// kChunk evaluations as an ordinary graph (no conditional node:
// the kernels return at once after the minimiser stopped)
int build_chunk_graph(OccState* st, int P, OccGraph& og) {
  cudaGraph_t g = nullptr;
  GB_TRY(gb::cuda_status(cudaGraphCreate(&g, 0), "occ chunk graph create"));
  auto fail = [&](cudaError_t e, const char* where) {
    cudaGraphDestroy(g);
    return gb::cuda_status(e, where);
  };
  cudaGraphNode_t prev = nullptr;
  for (int u = 0; u < kChunk; ++u) {
    cudaGraphNode_t n1 = nullptr;
    const cudaError_t e = add_eval_node(&n1, g, prev, st, P, 0, 0);
    if (e != cudaSuccess) return fail(e, "occ chunk graph: evaluation node");
    prev = n1;
  }
  cudaGraphExec_t exec = nullptr;
  cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
  if (e != cudaSuccess) return fail(e, "occ chunk graph: instantiate");
  og.chunk_graph = g;
  og.chunk_exec = exec;
  return GB_OK;
}

// The host-driven minimisation: init, then replays of the chunk graph until
// the phase copied back reads done (at most the evaluation cap's worth of
// replays), then the occupations and C^J, C^K.  The phase comes back through
// a stream-ordered copy to pageable memory (it returns once the replay has
// run), so nothing synchronises more than `s`.
int run_host_driven(OccState* st, const OccArgs& a, const OccGraph& og, cudaStream_t s, const char* name) {
  occ_init_kernel<<<1, kStepThreads, 0, s>>>(st, a);
  GB_CHECK_LAUNCH(name);
  const long long maxev = 1 + 200LL * (a.maxiter + 1);
  const long long max_replays = maxev / kChunk + 2;
  int phase = PH_INIT;
  for (long long r = 0; r < max_replays && phase != PH_DONE; ++r) {
    GB_TRY(gb::cuda_status(cudaGraphLaunch(og.chunk_exec, s), name));
    GB_TRY(gb::cuda_status(cudaMemcpyAsync(&phase, reinterpret_cast<const char*>(st) + offsetof(OccState, phase),
                                           sizeof(int), cudaMemcpyDeviceToHost, s),
                           name));
    GB_TRY(gb::cuda_status(cudaStreamSynchronize(s), name));
  }
  GB_REQUIRE(phase == PH_DONE, GB_ERR_TIMEOUT, "%s: the minimiser did not stop within the evaluation cap", name);
  occ_final_kernel<<<1, kStepThreads, 0, s>>>(st);
  GB_CHECK_LAUNCH(name);
  occ_cjck_kernel<<<kCjckCtas, kStepThreads, 0, s>>>(st);
  GB_CHECK_LAUNCH(name);
  return GB_OK;
}

int occ_run(const double* gamma0, const double* J, const double* K, const double* H, int nbf5, int no1, int ndoc,
            int ncwo, double gtol, int maxiter, int mode, double* gamma_out, double* grad_out, double* result,
            double* n_out, double* cj_out, double* ck_out, void* ws, size_t ws_bytes, void* stream,
            const char* name, bool host_driven = false) {
  gb::clear_error();
  GB_REQUIRE(gamma0 && J && K && H && result && ws, GB_ERR_INVALID_ARG, "%s: null pointer", name);
  GB_REQUIRE(mode == MODE_EVAL || gamma_out, GB_ERR_INVALID_ARG, "%s: null gamma_out", name);
  GB_REQUIRE((cj_out == nullptr) == (ck_out == nullptr), GB_ERR_INVALID_ARG, "%s: give both cj12 and ck12 or neither",
             name);
  GB_REQUIRE(no1 >= 0 && ndoc >= 1 && ncwo >= 1 && (long long)no1 + (long long)ndoc * (1 + ncwo) <= nbf5,
             GB_ERR_BAD_SHAPE, "%s: need no1 + ndoc (1 + ncwo) <= nbf5 (%d, %d, %d, %d)", name, no1, ndoc, ncwo,
             nbf5);
  GB_REQUIRE(maxiter >= 0 && gtol >= 0.0, GB_ERR_INVALID_ARG, "%s: need maxiter >= 0 and gtol >= 0", name);
  GB_REQUIRE(reinterpret_cast<uintptr_t>(ws) % 256 == 0, GB_ERR_INVALID_ARG, "%s: workspace not 256-byte aligned",
             name);
  gb::SizeCarve sc;
  OccState* dummy;
  OccArgs a{};
  occ_layout(sc, nbf5, ndoc, ncwo, &dummy, a);
  GB_REQUIRE(ws_bytes >= sc.used, GB_ERR_WORKSPACE, "%s: workspace of %zu bytes, need %zu", name, ws_bytes, sc.used);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  GB_TRY(gb::cuda_status(cudaStreamIsCapturing(s, &cs), name));
  GB_REQUIRE(cs == cudaStreamCaptureStatusNone, GB_ERR_UNSUPPORTED, "%s: not capturable (runs its own graph)", name);
  gb::Carve c(ws, ws_bytes);
  OccState* st = nullptr;
  occ_layout(c, nbf5, ndoc, ncwo, &st, a);
  a.J = J;
  a.K = K;
  a.H = H;
  a.gamma0 = gamma0;
  a.gamma_out = gamma_out ? gamma_out : a.stage;  // (an evaluation: x itself)
  a.grad_out = grad_out;
  a.res = result;
  a.n_out = n_out;
  a.cj_out = cj_out;
  a.ck_out = ck_out;
  a.P = nbf5;
  a.no1 = no1;
  a.ndoc = ndoc;
  a.ncwo = ncwo;
  a.maxiter = maxiter;
  a.mode = mode;
  a.gtol = gtol;
  std::unique_lock<std::mutex> lk(g_mu);
  const auto key = std::make_tuple(gb::current_context_id(), (const void*)ws, nbf5);
  auto it = g_graphs.find(key);
  if (it == g_graphs.end()) {
    OccGraph og;
    GB_TRY(build_graph(st, nbf5, og));
    it = g_graphs.emplace(key, og).first;
  }
  if (host_driven) {
    if (!it->second.chunk_exec) GB_TRY(build_chunk_graph(st, nbf5, it->second));
    // the replay loop runs without the cache lock (other workspaces' calls
    // proceed meanwhile); this workspace's entry stays until gb_occ_release,
    // which must not overlap a call on the same workspace
    const OccGraph og = it->second;
    lk.unlock();
    const int pi = gb::prof_begin(name, s);
    const int rc = run_host_driven(st, a, og, s, name);
    gb::prof_end(pi, s);
    return rc;
  }
  void* ip[] = {&st, &a};
  cudaKernelNodeParams kp{};
  kp.func = (void*)occ_init_kernel;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(kStepThreads);
  kp.kernelParams = ip;
  GB_TRY(gb::cuda_status(cudaGraphExecKernelNodeSetParams(it->second.exec, it->second.init, &kp), name));
  const int pi = gb::prof_begin(name, s);
  const cudaError_t e = cudaGraphLaunch(it->second.exec, s);
  gb::prof_end(pi, s);
  return gb::cuda_status(e, name);
}

}  // namespace

extern "C" size_t gb_occ_workspace_bytes(int nbf5, int ndoc, int ncwo) {
  if (nbf5 < 1 || ndoc < 1 || ncwo < 1) return 0;
  gb::SizeCarve sc;
  OccState* st;
  OccArgs a{};
  occ_layout(sc, nbf5, ndoc, ncwo, &st, a);
  return sc.used;
}

extern "C" int gb_occ_minimize_dev(const double* gamma0, const double* J_MO, const double* K_MO,
                                   const double* H_core, int nbf5, int no1, int ndoc, int ncwo, double gtol,
                                   int maxiter, double* gamma_out, double* result, double* n_out, double* cj12_out,
                                   double* ck12_out, void* ws, size_t ws_bytes, void* stream) {
  return occ_run(gamma0, J_MO, K_MO, H_core, nbf5, no1, ndoc, ncwo, gtol, maxiter, MODE_MIN, gamma_out, nullptr,
                 result, n_out, cj12_out, ck12_out, ws, ws_bytes, stream, "gb_occ_minimize_dev");
}

extern "C" int gb_occ_minimize_dev_sync(const double* gamma0, const double* J_MO, const double* K_MO,
                                        const double* H_core, int nbf5, int no1, int ndoc, int ncwo, double gtol,
                                        int maxiter, double* gamma_out, double* result, double* n_out,
                                        double* cj12_out, double* ck12_out, void* ws, size_t ws_bytes, void* stream) {
  return occ_run(gamma0, J_MO, K_MO, H_core, nbf5, no1, ndoc, ncwo, gtol, maxiter, MODE_MIN, gamma_out, nullptr,
                 result, n_out, cj12_out, ck12_out, ws, ws_bytes, stream, "gb_occ_minimize_dev_sync", true);
}

extern "C" int gb_occ_energy_grad_dev(const double* gamma, const double* J_MO, const double* K_MO,
                                      const double* H_core, int nbf5, int no1, int ndoc, int ncwo, double* result,
                                      double* grad, void* ws, size_t ws_bytes, void* stream) {
  return occ_run(gamma, J_MO, K_MO, H_core, nbf5, no1, ndoc, ncwo, 0.0, 0, MODE_EVAL, nullptr, grad, result,
                 nullptr, nullptr, nullptr, ws, ws_bytes, stream, "gb_occ_energy_grad_dev");
}

extern "C" int gb_occ_release(const void* ws) {
  gb::clear_error();
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto it = g_graphs.begin(); it != g_graphs.end();) {
    if (std::get<1>(it->first) == ws) {
      cudaGraphExecDestroy(it->second.exec);
      cudaGraphDestroy(it->second.graph);
      if (it->second.chunk_exec) cudaGraphExecDestroy(it->second.chunk_exec);
      if (it->second.chunk_graph) cudaGraphDestroy(it->second.chunk_graph);
      it = g_graphs.erase(it);
    } else {
      ++it;
    }
  }
  return GB_OK;
}
