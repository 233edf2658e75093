// The reduced iteration: BiCGSTAB without the rows of color 0.
//
// Color 0 is eliminated first, so its rows of L are the identity and its rows
// of U are A's, and the same holds for U^T, L^T and A^T. Hence
// (A M^-1 p)_0 = (M M^-1 p)_0 = p_0: on the rows of color 0 (the head, about
// half of all rows on a grid) v = p and t = s, without any product. By
// induction every vector of the iteration is, on the head, a number times the
// initial residual r0:
//
//   p = cp r0,  v = p,  s = cs r0 with cs = cr - alpha cp,  t = s,
//   r = cr r0 with cr = (1 - omega) cs,  cp' = cr + beta (1 - omega) cp,
//
// its share of each dot product is a product of these numbers with ||r0||^2
// (Ctl::head_rr), and the head's part of the first sweep on the other rows
// (the tail), sum_j L_ij p_j, is cp g with g = L_i0 r0 formed once a solve.
// What is left of one preconditioned product is
//
//   tail, first sweep:  y = p - cp g (- the few L blocks inside the tail);
//                       the rows of color 1 have none, so the kernel that
//                       writes p (or s) also writes their y and D^-1 y;
//   small steps:        the tail's other colors, both sweeps;
//   head, second sweep: p^ = D^-1 (cp r0 - sum U p^);
//   SpMV of the tail:   v = A p^, (v, rt);
//
// i.e. half of the blocks of A, the head's half of U and two diagonals
// instead of A, L, U and D: 0.71 instead of 1.30 GB an iteration on the
// 500k-cell system in FP64, the vectors included. x is advanced on the tail alone; at the end the
// head's equations give its x from the residual they are left with,
// x_0 = A_00^-1 (b_0 - cr r0 - sum A_0j x_j). In exact arithmetic the
// iterates, norms and stop tests are those of the full iteration; rounding
// adds what the head's blocks make of theirs, so that a factorization with
// ill-conditioned ones keeps the full iteration (reduced_run). (With U^T, L^T
// and A^T for the adjoint: base0 = D^-T r0, g = U_i0^T base0, head:
// p^ = cp base0 - sum L^T p^.)
//
// base holds, in one vector, r0 (adjoint: D^-T r0) on the head and -g on the
// tail, so a head row's own value is coef * base and a tail row's is
// src + coef * base with coef = cp (src = p) or cs (src = s).
#pragma once

#include "gbilu_kernels.cuh"

namespace gbilu {

// The tail's rows and what the first sweep's step of color 1 needs. Rows are
// counted from the first row of the tail; color 1 comes first.
template <typename V, typename T> struct Tail {
  int row0;             // first row of the tail (rows of color 0 before it)
  int rows;             // rows of the tail
  int rows1;            // rows of color 1
  int split1;           // its leading rows with a neighbour of a higher color
  int slice1;           // its first slice
  int d_first;          // adjoint: D^-T in the first sweep; else D^-1 in the second
  const V *dmat;
  const T *base;
  T *ybuf, *hat;
};

// The first sweep of tail row t (counted from row0) with own value w + coef
// * base: color 1 is stored as its step says; the rows of the later colors,
// which the apply's small steps compute, get the sentinel that those steps'
// consumers wait on. (a: base of the row.)
template <typename V, typename T>
__device__ __forceinline__ void tail_first(const Tail<V, T> &P, int t, T coef, T b0, T b1, T b2,
                                           T w0, T w1, T w2) {
  const int i = 3 * (P.row0 + t);
  const T sent = sentinel_value<T>();
  if (t >= P.rows1) {
    P.ybuf[i] = sent; P.ybuf[i + 1] = sent; P.ybuf[i + 2] = sent;
    P.hat[i] = sent; P.hat[i + 1] = sent; P.hat[i + 2] = sent;
    return;
  }
  T a0 = fma(coef, b0, w0), a1 = fma(coef, b1, w1), a2 = fma(coef, b2, w2);
  const bool split = t < P.split1;
  if (P.d_first || !split)
    apply_dp<V, T, true>(P.dmat + (size_t)(P.slice1 + (t >> 5)) * 9 * 32, t & 31, a0, a1, a2);
  T *out = P.hat + i;
  if (split) {
    out = P.ybuf + i;
    P.hat[i] = sent; P.hat[i + 1] = sent; P.hat[i + 2] = sent;
  }
  out[0] = a0; out[1] = a1; out[2] = a2;
}

// base0 = D^-T r0 on the head (adjoint), in place.
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_base_head(const Ctl *ctl, int rows, const V *__restrict__ dmat, T *__restrict__ base) {
  if (ctl->done) return;
  const int t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= rows) return;
  T a0 = base[3 * t], a1 = base[3 * t + 1], a2 = base[3 * t + 2];
  apply_dp<V, T, true>(dmat + (size_t)(t >> 5) * 9 * 32, t & 31, a0, a1, a2);
  base[3 * t] = a0; base[3 * t + 1] = a1; base[3 * t + 2] = a2;
}

// base = -g on the tail, from the head's columns of the full first-sweep
// matrix (a row's first blocks: columns ascend by color), and the first
// sweep of the solve's first apply (p = r0, cp = 1). One warp a slice.
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_base_tail(const Ctl *ctl, Tail<V, T> P, int S, const int2 *__restrict__ srows,
            const int *__restrict__ off, const int *__restrict__ col, const V *__restrict__ val,
            const T *__restrict__ p, T *base, T *sh, T *ysh) {
  if (ctl->done) return;
  const int lane = threadIdx.x & 31;
  for (int s = P.slice1 + blockIdx.x * kWarps + (threadIdx.x >> 5); s < S; s += gridDim.x * kWarps) {
    const int2 sr = srows[s];
    if (lane >= sr.y) continue;
    const int row = sr.x + lane;
    const int o = off[s], w = off[s + 1] - o;
    T a0 = 0, a1 = 0, a2 = 0;
    for (int k = 0; k < w; ++k) {
      const int c = ldg_stream(col + (size_t)(o + k) * 32 + lane);
      if (c < 0 || c >= P.row0) break;   // padding, or the first block inside the tail
      V b[9];
      load_block<V, true>(val + (size_t)(o + k) * 9 * 32, lane, b);
      const T *xs = base + 3 * c;
      const T x0 = xs[0], x1 = xs[1], x2 = xs[2];
      a0 = fma(-(T)b[0], x0, a0); a0 = fma(-(T)b[1], x1, a0); a0 = fma(-(T)b[2], x2, a0);
      a1 = fma(-(T)b[3], x0, a1); a1 = fma(-(T)b[4], x1, a1); a1 = fma(-(T)b[5], x2, a1);
      a2 = fma(-(T)b[6], x0, a2); a2 = fma(-(T)b[7], x1, a2); a2 = fma(-(T)b[8], x2, a2);
    }
    base[3 * row] = a0; base[3 * row + 1] = a1; base[3 * row + 2] = a2;
    tail_first(P, row - P.row0, (T)1, a0, a1, a2, p[3 * row], p[3 * row + 1], p[3 * row + 2]);
    // what the small steps of the first s write or wait for (k_tail_flow)
    const int t = row - P.row0;
    if (sh && (t < P.split1 || t >= P.rows1)) {
      const T sent = sentinel_value<T>();
      for (int e = 0; e < 3; ++e) { sh[3 * row + e] = sent; ysh[3 * row + e] = sent; }
    }
  }
}

// The vector kernels deal their warps' groups of 32 rows to the CTAs in turn,
// so that the groups of a last, partial round spread over all SMs.
__device__ __forceinline__ int first_row() {
  return 32 * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) + (threadIdx.x & 31);
}

// Steps 6-8 on the tail (k_update_s) and the first sweep of the next apply:
// s = r - alpha v, ||s|| and the stop tests; y or hat of color 1 from s.
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_tail_s(Ctl *ctl, Tail<V, T> P, const T *__restrict__ r, const T *__restrict__ v,
         T *__restrict__ s, double *partials) {
  if (ctl->done) return;
  const T alpha = (T)ctl->alpha, cs = (T)ctl->cs;
  double d = 0.0;
  DF f = {0.f, 0.f};
  for (int t = first_row(); t < P.rows; t += gridDim.x * kThreads) {
    const int i = 3 * (P.row0 + t);
    const T *b = P.base + i;
    const T b0 = b[0], b1 = b[1], b2 = b[2];
    const T s0 = fma(-alpha, v[i], r[i]), s1 = fma(-alpha, v[i + 1], r[i + 1]),
            s2 = fma(-alpha, v[i + 2], r[i + 2]);
    s[i] = s0; s[i + 1] = s1; s[i + 2] = s2;
    if (sizeof(T) == 8) {
      d += (double)s0 * s0 + (double)s1 * s1 + (double)s2 * s2;
    } else {
      df_add_prod(f, (float)s0, (float)s0); df_add_prod(f, (float)s1, (float)s1);
      df_add_prod(f, (float)s2, (float)s2);
    }
    tail_first(P, t, cs, b0, b1, b2, s0, s1, s2);
  }
  if (sizeof(T) == 4) d = df_value(f);
  double vv[1] = {d}, tot[1];
  if (grid_sum<1>(vv, partials, &ctl->counter[3], tot) && threadIdx.x == 0) finish_s(ctl, tot[0]);
}

// Steps 15-17 on the tail (k_update_p) and the first sweep of the next
// apply. Also drives the graph's while loop.
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_tail_p(Ctl *ctl, Tail<V, T> P, const T *__restrict__ r, const T *__restrict__ v,
         T *__restrict__ p, T *__restrict__ rt, unsigned long long cond) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->body_runs += 1;
    // hard stop as a second guard: the loop can never run past maxit + 1
    if (cond)
      cudaGraphSetConditional((cudaGraphConditionalHandle)cond,
                              (ctl->done || ctl->body_runs > ctl->maxit + 1) ? 0u : 1u);
  }
  if (ctl->done) return;
  const T beta = (T)ctl->beta, omega = (T)ctl->omega, cp = (T)ctl->cp;
  const bool restart = ctl->restart;
  for (int t = first_row(); t < P.rows; t += gridDim.x * kThreads) {
    const int i = 3 * (P.row0 + t);
    const T *b = P.base + i;
    const T b0 = b[0], b1 = b[1], b2 = b[2];
    const T r0 = r[i], r1 = r[i + 1], r2 = r[i + 2];
    const T p0 = fma(beta, fma(-omega, v[i], p[i]), r0),
            p1 = fma(beta, fma(-omega, v[i + 1], p[i + 1]), r1),
            p2 = fma(beta, fma(-omega, v[i + 2], p[i + 2]), r2);
    if (restart) { rt[i] = r0; rt[i + 1] = r1; rt[i + 2] = r2; }
    p[i] = p0; p[i + 1] = p1; p[i + 2] = p2;
    tail_first(P, t, cp, b0, b1, b2, p0, p1, p2);
  }
}

// --------------------------------------------------------------------------
// the vector kernels with the small steps beside them (FP64, three and more
// colors)
// --------------------------------------------------------------------------

// What a tail kernel needs to run the small steps too.
struct Flow {
  const int *off1r, *col1r; const double *val1r;   // first sweep, the tail's columns
  const int *off2, *col2; const double *val2;      // second sweep
  int groups;             // groups of three warps on the small steps
};
constexpr int kFlowThreads = 512;
constexpr int kFlowWarps = kFlowThreads / 32;
constexpr int kFlowGroups = 4;     // at most: the other warps form p or s

// Component c of a row: a - its blocks' row c times x, once every value is
// there (sentinels in x are waited for; a wait that runs out stops the solve).
__device__ __forceinline__ double flow_row(const double *__restrict__ sv,
                                           const int *__restrict__ sc, int w, int lane, int c,
                                           const double *x, double a, Ctl *ctl) {
  constexpr int B = 2;   // (4: 2 % slower)
  for (int k0 = 0; k0 < w; k0 += B) {
    int cc[B];
    double y[B][3];
    double b[B][3];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      cc[j] = k0 + j < w ? sc[(k0 + j) * 32 + lane] : -1;
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (k0 + j < w) b[j][e] = sv[(size_t)(k0 + j) * 288 + sl_idx<double>(0, 3 * c + e, lane)];
    }
    unsigned int spins = 0;
    bool wait;
    do {
      const double *miss = nullptr;
#pragma unroll
      for (int j = 0; j < B; ++j)
        if (cc[j] >= 0) {
          const double *xs = x + 3 * cc[j];
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            y[j][e] = ld_relaxed(xs + e);
            if (is_sentinel(y[j][e])) miss = xs + e;
          }
        }
      wait = miss != nullptr;
      // one missing value is watched, then all are loaded again (watching all
      // of them crowds out the stores that they wait for)
      while (wait && is_sentinel(ld_relaxed(miss))) wait = poll_again(ctl, spins);
    } while (wait);
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (cc[j] >= 0)
#pragma unroll
        for (int e = 0; e < 3; ++e) a = fma(-b[j][e], y[j][e], a);
  }
  return a;
}

// k_tail_s and k_tail_p (MODE 1, 2; 0: p is there, the small steps alone) for
// three and more colors: while most warps form s or p and color 1's first
// sweep, a few run the small colors' steps of the next apply, ordered by
// their data: their results (hat of color 1's split rows and of the later
// colors) and y were preset to the sentinel by k_update_r, split rows come
// first among color 1's, and a consumer loads again until a value is there.
// A step reads only rows of earlier steps and of warps that wait for nothing,
// every group takes its slices in step order, and the launch is cooperative:
// every wait ends. (In the apply's launch, before the head's step and a grid
// barrier, the small steps of a 500k-cell system with five colors kept the GPU
// waiting for 17 us an apply in FP64, and FP64's few warps cannot hide them
// there.) Measured, vector kernel + apply with 475,000 rows: s 16.4 + 52.5 ->
// 24.6 + 34.4 us, p 12.3 + 52.5 -> 20.7 + 34.4; an iteration 238 -> 219, with
// 209,000 rows 149 -> 126. In FP32 the small steps cost less, and a cooperative
// vector kernel with fewer warps takes as much more: s 11.2 + 24.8 against 20.9
// + 14.8 us, an iteration 200 against 208. There they stay in the apply's
// launch (k_ilu_coop).
template <int MODE>
__global__ void __launch_bounds__(kFlowThreads, 1)
k_tail_flow(Ctl *ctl, Tail<double, double> P, Flow F, const __grid_constant__ PhaseList ph,
            const double *__restrict__ r, const double *__restrict__ v, double *w, double *rt,
            double *partials, unsigned long long cond) {
  using V = double;
  using T = double;
  __shared__ T xch[kFlowGroups][3][32];
  __shared__ double red[kFlowThreads];
  __shared__ bool last;
  if (MODE == 2 && blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->body_runs += 1;
    // hard stop as a second guard: the loop can never run past maxit + 1
    if (cond)
      cudaGraphSetConditional((cudaGraphConditionalHandle)cond,
                              (ctl->done || ctl->body_runs > ctl->maxit + 1) ? 0u : 1u);
  }
  if (ctl->done) return;
  const T alpha = (T)ctl->alpha, beta = (T)ctl->beta, omega = (T)ctl->omega;
  const T coef = (T)(MODE == 1 ? ctl->cs : ctl->cp);
  const bool restart = MODE == 2 && ctl->restart;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, G = gridDim.x, bid = blockIdx.x;
  const int w0 = 3 * F.groups;
  double d = 0.0;
  auto updated = [&](int i) -> T {   // the new s or p at entry i
    if (MODE == 0) return w[i];
    const T ri = r[i];
    const T x = MODE == 1 ? fma(-alpha, v[i], ri) : fma(beta, fma(-omega, v[i], w[i]), ri);
    w[i] = x;
    if (MODE == 2 && restart) rt[i] = ri;
    if (MODE == 1) d = fma(x, x, d);
    return x;
  };
  if (warp < w0) {
    // slice s of a step belongs to CTA s % G; three warps, one per component
    const int g = warp / 3, c = warp % 3;
    T(&xg)[3][32] = xch[g];
    auto times_d = [&](const V *dm, T a) -> T {
      xg[c][lane] = a;
      group_sync(g);
      const T z = dot3<T>((T)dm[sl_idx<V>(0, 3 * c, lane)], (T)dm[sl_idx<V>(0, 3 * c + 1, lane)],
                          (T)dm[sl_idx<V>(0, 3 * c + 2, lane)], xg[0][lane], xg[1][lane],
                          xg[2][lane]);
      group_sync(g);
      return z;
    };
    T *y = P.ybuf, *hat = P.hat;
    for (int q = 0; q + 1 < ph.n; ++q) {
      const Phase &S = ph.p[q];
      const int *off = S.mat ? F.off2 : F.off1r, *col = S.mat ? F.col2 : F.col1r;
      const V *val = S.mat ? F.val2 : F.val1r;
      const int end = S.slice0 + ((S.nrows + 31) >> 5);
      int s = S.slice0 + ((bid - S.slice0) % G + G) % G;   // the CTA's first slice of the step
      for (s += g * G; s < end; s += F.groups * G) {
        const int rr = 32 * (s - S.slice0) + lane, row = S.row0 + rr, e = 3 * row + c;
        const bool act = rr < S.nrows;
        const V *dm = P.dmat + (size_t)s * 288;
        const int o = off[s], wd = off[s + 1] - o;
        T a = 0;
        if (act) {
          if (S.own_y) {
            unsigned int spins = 0;
            while (is_sentinel(a = ld_relaxed(y + e)) && poll_again(ctl, spins)) {}
          } else {   // a row of color 2 and up gets its p or s here
            a = updated(e);
            a = fma(coef, P.base[e], a);
          }
          a = flow_row(val + (size_t)o * 288, col + (size_t)o * 32, wd, lane, c,
                             S.nbr_hat ? hat : y, a, ctl);
        }
        if (S.has_d) a = times_d(dm, a);
        bool fin = true;
        if (S.to_y) {
          fin = row >= S.final0;
          if (act && !fin) st_relaxed(y + e, a);
          if (S.final_d) a = times_d(dm, a);
        }
        if (act && fin) st_relaxed(hat + e, a);
      }
    }
  } else if (MODE != 0) {
    // color 1, groups of 32 rows dealt to the CTAs in turn
    for (int j = (warp - w0) * G + bid; 32 * j < P.rows1; j += (kFlowWarps - w0) * G) {
      const int t = 32 * j + lane;
      if (t >= P.rows1) continue;
      const int i = 3 * (P.row0 + t);
      const T b0 = P.base[i], b1 = P.base[i + 1], b2 = P.base[i + 2];
      const T x0 = updated(i), x1 = updated(i + 1), x2 = updated(i + 2);
      T a0 = fma(coef, b0, x0), a1 = fma(coef, b1, x1), a2 = fma(coef, b2, x2);
      const bool split = t < P.split1;
      if (P.d_first || !split)
        apply_dp<V, T, true>(P.dmat + (size_t)(P.slice1 + j) * 288, lane, a0, a1, a2);
      T *out = (split ? P.ybuf : P.hat) + i;
      if (split) {
        st_relaxed(out, a0); st_relaxed(out + 1, a1); st_relaxed(out + 2, a2);
      } else {
        out[0] = a0; out[1] = a1; out[2] = a2;
      }
    }
  }
  if (MODE != 1) return;
  // ||s||^2: the CTA's sum, then the CTAs' by the last one, in a fixed order
  const int t = threadIdx.x;
  red[t] = d;
  __syncthreads();
  double x = 0.0;
  if (t < 128) x = (red[t] + red[t + 128]) + (red[t + 256] + red[t + 384]);
  __syncthreads();
  if (t < 128) red[t] = x;
  __syncthreads();
  if (t >= 32) return;
  x = (red[t] + red[t + 32]) + (red[t + 64] + red[t + 96]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (t == 0) {
    partials[bid] = x;
    unsigned int prev;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(prev) : "l"(&ctl->counter[3]) : "memory");
    last = prev == gridDim.x - 1;
  }
  __syncwarp();
  if (!last) return;
  x = 0.0;
  for (int b = t; b < G; b += 32) x += __ldcg(partials + b);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (t == 0) {
    ctl->counter[3] = 0u;
    finish_s(ctl, x);
  }
}

// The head's x after the loop, from its equations and the residual they are
// left with: forward x = D^-1 (b - c r0 - sum U x), adjoint
// x = D^-T (b - c r0) - sum L^T x, c = cs after a stop in a first half, else
// cr. x keeps its start value when no iteration moved it (zero in a
// refinement step, which then adds nothing).
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_finish_head(const Ctl *ctl, int rows, int d_first, const int *__restrict__ off,
              const int *__restrict__ col, const V *__restrict__ val, const V *__restrict__ dmat,
              const T *__restrict__ b, const T *__restrict__ r0, T *x, Refine out) {
  if (ctl->half < 0 || !(ctl->stop_half || ctl->x_moved)) return;
  const int t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= rows) return;
  const T c = (T)(ctl->stop_half ? ctl->cs : ctl->cr);
  const int s = t >> 5, lane = t & 31;
  const V *d = dmat + (size_t)s * 9 * 32;
  T a0 = fma(-c, r0[3 * t], b[3 * t]), a1 = fma(-c, r0[3 * t + 1], b[3 * t + 1]),
    a2 = fma(-c, r0[3 * t + 2], b[3 * t + 2]);
  if (d_first) apply_dp<V, T, true>(d, lane, a0, a1, a2);
  const int o = off[s];
  row_blocks<V, T, true, false, true>(col, val, o, off[s + 1] - o, lane, x, x, 0, a0, a1, a2);
  if (!d_first) apply_dp<V, T, true>(d, lane, a0, a1, a2);
  x[3 * t] = a0; x[3 * t + 1] = a1; x[3 * t + 2] = a2;
  if (out.x64 && ctl->status != ST_BREAKDOWN && ctl->status != ST_NONFINITE) {
    double *y = out.x64 + 3 * t;
    y[0] = fma(out.scale, (double)a0, y[0]);
    y[1] = fma(out.scale, (double)a1, y[1]);
    y[2] = fma(out.scale, (double)a2, y[2]);
  }
}

}  // namespace gbilu
