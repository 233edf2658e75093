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
// instead of A, L, U and D: 0.55 instead of 1.30 GB an iteration on the
// 500k-cell system in FP64. x is advanced on the tail alone; at the end the
// head's equations give its x from the residual they are left with,
// x_0 = A_00^-1 (b_0 - cr r0 - sum A_0j x_j). All of this is exact: the
// iterates, norms and stop tests are those of the full iteration up to
// rounding. (With U^T, L^T and A^T for the adjoint: base0 = D^-T r0,
// g = U_i0^T base0, head: p^ = cp base0 - sum L^T p^.)
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
            const T *__restrict__ p, T *base) {
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

// The head's x after the loop, from its equations and the residual they are
// left with: forward x = D^-1 (b - c r0 - sum U x), adjoint
// x = D^-T (b - c r0) - sum L^T x, c = cs after a stop in a first half, else
// cr. x keeps its start value when no iteration moved it.
template <typename V, typename T>
__global__ void __launch_bounds__(kThreads)
k_finish_head(const Ctl *ctl, int rows, int d_first, const int *__restrict__ off,
              const int *__restrict__ col, const V *__restrict__ val, const V *__restrict__ dmat,
              const T *__restrict__ b, const T *__restrict__ r0, T *x) {
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
}

}  // namespace gbilu
