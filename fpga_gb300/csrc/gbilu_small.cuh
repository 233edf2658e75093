// A whole reduced solve (gbilu_reduced.cuh) in one cooperative launch, for
// systems that one wave of CTAs holds.
//
// What bounds such a system is not work but latency: seven kernels an
// iteration, each a launch, a few dependent loads, a serial chain of FP64
// instructions (65 cycles each; a warp issues one every 64) and a grid
// reduction, 8-9 us apiece for 4,000 cells. Here one CTA per SM keeps its
// slices' blocks, column indices and diagonal inverses in shared memory for
// the whole solve (bulk copies when the launch starts; what does not fit is
// read from L2), three warps share a slice, one per component, so the FP64
// chain is a third, all gathers of a row are in flight together, a vector
// entry belongs to one thread for the whole solve, and a step boundary is a
// grid barrier (about 1.5 us) instead of a kernel boundary. ||s|| is summed
// with the reduction after it, so a stop in a first half has run the second
// SpMV in vain. b and x are read and written in the caller's numbering by the
// same launch.
//
// Measured against the separate kernels (solves to 1e-8, start and end
// included): an iteration of 33,000 rows (three colors) 78 -> 49 us, of 59,000
// 73 -> 49, of 108,000 86 -> 67; one_launch_size has more and where it ends.
// It holds every SM until it ends (gbilu_options.one_launch). Ordering the steps between two
// reductions by their data instead (results preset to a sentinel, consumers
// polling) gave 28.7 us for 4,000 cells with two colors, but 47 instead of 44
// with three and 75 instead of 53 for 33,000 cells: polled loads bypass L1.
//
// Per row and component the arithmetic is that of the separate kernels;
// dot products are summed in this kernel's own fixed order. The scalars are
// computed by every CTA from the same totals (CTA-local copy of Ctl), so all
// CTAs take the same decisions.
#pragma once

#include "gbilu_reduced.cuh"

namespace gbilu {

constexpr int kSmallThreads = 384;
constexpr int kSmallGroups = kSmallThreads / 32 / 3;   // three warps a slice
static_assert(kSmallThreads == 3 * 128, "the sums add three values a thread");
constexpr int kSmallOwn = 64;                          // slices of a CTA

// FP64 (T = double): solves A x = b from x, both in the input numbering.
// FP32 (T = float), an inner solve of the mixed form: A d = scale * r64 from
// d = 0, then x64 += unscale * d (device numbering).
template <typename V, typename T> struct SmallArgs {
  Ctl *host_ctl;                  // the final state (mapped host memory)
  int *fail, *host_fail;          // the kind of a failed wait (see give_up): for the
                                  // other CTAs, and for the host (mapped); 0 before
  unsigned long long *bar;        // barrier counter: a multiple of arrivals
  unsigned int arrivals;          // CTAs that a barrier waits for: the grid
  unsigned int spins;             // polls after which a wait gives up
  int *x_nonzero;                 // 0 between launches
  double *partials;               // 9 sums a CTA
  const int2 *srows;
  int S, S0, S1;                  // slices; the first of the tail, of color 2
  int n0, split1;                 // head rows; Tail's split1
  int transpose;
  const int *offA, *colA; const V *valA;
  const int *off1, *col1; const V *val1;
  const int *off1r, *col1r; const V *val1r;
  const int *off2, *col2; const V *val2;
  const V *dmat;
  T *b, *x, *r, *rt, *p, *ph, *v, *s, *sh, *t, *y, *base;
  const int *perm;                // device row -> input row
  const double *b_in;
  double *x_io;
  bool from_zero;                 // x0 = 0: x_io is only written
  const double *r64;
  double *x64;
  double scale, unscale;          // 1 / ||r64||, ||r64||
  double tol;
  int absolute, maxit;
  unsigned long long timeout_ns;
  int smem_bytes;                 // dynamic shared memory
};

// Shared state of a CTA.
template <typename V, typename T> struct SmallCta {
  Ctl c;
  uint64_t copies;                // mbarrier of the bulk copies
  int pos[kSmallOwn], w[kSmallOwn], o[kSmallOwn];   // place (-1: L2), width, first slot
  int2 rows[kSmallOwn];
  double red[3][kSmallThreads], tot[3];
  T xch[kSmallGroups][3][32];
  int ok;
};

// Component c of one row: a -+ sum over its blocks' row c times x (other SMs
// wrote it in this launch, before a grid barrier, whose acquire makes L1 loads
// see it). Columns ascend; those from limit on end the row, as padding does.
// The gathers of B blocks go out together: FP64 3 (an iteration of 108,000
// cells 63 us; with 2 63, 4 66, 5 72, 8 71), FP32 8 (74; 3 to 6: 75-79). (Not
// inlined: its sites would spill each other.)
template <typename V, typename T, bool NEG>
__device__ __noinline__ T comp_row(const V *sv, const int *sc, int w, int lane, int c, const T *x,
                                   int limit, T a) {
  constexpr int B = sizeof(T) == 8 ? 3 : 8;
  for (int k0 = 0; k0 < w; k0 += B) {
    int cc[B];
    T y[B][3];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      cc[j] = k0 + j < w ? sc[(k0 + j) * 32 + lane] : -1;
      if (cc[j] >= limit) cc[j] = -1;
    }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (cc[j] >= 0) {
        const T *xs = x + 3 * cc[j];
#pragma unroll
        for (int e = 0; e < 3; ++e) y[j][e] = xs[e];
      }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (cc[j] >= 0) {
        const V *b = sv + (size_t)(k0 + j) * 9 * 32;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const T be = (T)b[sl_idx<V>(0, 3 * c + e, lane)];
          a = fma(NEG ? -be : be, y[j][e], a);
        }
      }
    if (cc[B - 1] < 0) break;
  }
  return a;
}

// The three components of a group's rows meet: component c of D a. Every
// warp of the group takes part.
template <typename V, typename T>
__device__ __forceinline__ T comp_d(T (&xch)[3][32], int grp, int c, int lane, const V *d, T a) {
  xch[c][lane] = a;
  group_sync(grp);
  const T z = dot3<T>((T)d[sl_idx<V>(0, 3 * c, lane)], (T)d[sl_idx<V>(0, 3 * c + 1, lane)],
                      (T)d[sl_idx<V>(0, 3 * c + 2, lane)], xch[0][lane], xch[1][lane],
                      xch[2][lane]);
  group_sync(grp);
  return z;
}

template <typename V, typename T> struct SmallSolve {
  const SmallArgs<V, T> &A;
  SmallCta<V, T> &S;
  unsigned char *mem;
  const int G, bid, grp, c, lane;
  int own, tail0;                 // this CTA's slices; its first tail slice
  bool late = false;              // this thread's wait for the copies ran out
  bool failed = false;

  __device__ SmallSolve(const SmallArgs<V, T> &a, SmallCta<V, T> &s, unsigned char *m)
      : A(a), S(s), mem(m), G(gridDim.x), bid(blockIdx.x), grp((threadIdx.x >> 5) / 3),
        c((threadIdx.x >> 5) % 3), lane(threadIdx.x & 31) {
    own = (A.S - bid + G - 1) / G;
    tail0 = A.S0 > bid ? (A.S0 - bid + G - 1) / G : 0;
  }

  // own slice i is slice bid + i * G; the groups take the slices in turn
  __device__ int slice(int i) const { return bid + i * G; }
  template <typename F> __device__ __forceinline__ void each(int i0, int i1, F f) const {
    if (grp < kSmallGroups)
      for (int i = i0 + grp; i < i1; i += kSmallGroups) {
        const int2 sr = S.rows[i];
        f(i, lane < sr.y, sr.x + lane);
      }
  }
  template <typename F> __device__ __forceinline__ void head(F f) const { each(0, tail0, f); }
  template <typename F> __device__ __forceinline__ void tail(F f) const { each(tail0, own, f); }

  // the slice's blocks in the matrix of its steps (head: U or L^T, tail: A)
  __device__ const V *vals(int i) const {
    if (S.pos[i] >= 0) return reinterpret_cast<const V *>(mem + S.pos[i]);
    return (i < tail0 ? A.val2 : A.valA) + (size_t)S.o[i] * 9 * 32;
  }
  __device__ const int *cols(int i) const {
    if (S.pos[i] >= 0)
      return reinterpret_cast<const int *>(mem + S.pos[i] + (size_t)S.w[i] * 9 * 32 * sizeof(V));
    return (i < tail0 ? A.col2 : A.colA) + (size_t)S.o[i] * 32;
  }
  // whether the slice's steps apply D (head: the second sweep's; tail: color 1)
  __device__ bool uses_d(int i) const { return i < tail0 ? !A.transpose : slice(i) < A.S1; }
  __device__ const V *dblk(int i) const {
    if (S.pos[i] >= 0 && uses_d(i))
      return reinterpret_cast<const V *>(mem + S.pos[i] +
                                         (size_t)S.w[i] * (9 * 32 * sizeof(V) + 32 * sizeof(int)));
    return A.dmat + (size_t)slice(i) * 9 * 32;
  }

  // A wait ran out (1: of a barrier, 2: of the copies): the first kind is kept.
  // The host learns of it from the CTA that gave up itself: CTA 0 may have
  // passed the last barrier by then.
  __device__ void give_up(int kind) {
    const int first = atomicCAS(A.fail, 0, kind);
    *(volatile int *)A.host_fail = first ? first : kind;
    __threadfence_system();
  }

  // Grid barrier; the counter only grows, 64 bits wide, and every launch adds
  // a multiple of its grid. Bounded; a wait that ran out, here or before
  // (late), fails the run in every CTA.
  __device__ bool barrier() {
    const int any_late = __syncthreads_or(late);
    if (threadIdx.x == 0) {
      S.ok = !any_late;
      if (any_late) give_up(2);
      unsigned long long ticket, now;
      asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;"
                   : "=l"(ticket) : "l"(A.bar), "l"(1ull) : "memory");
      const unsigned long long target = (ticket / A.arrivals + 1) * A.arrivals;
      unsigned int spins = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(A.bar) : "memory");
        if (now >= target) break;
        if (++spins > A.spins || ((spins & 1023) == 0 && *(volatile int *)A.fail)) {
          S.ok = 0;
          give_up(1);
          break;
        }
        if (spins > 256) __nanosleep(32);
      }
    }
    __syncthreads();
    if (!S.ok) failed = true;
    return !failed;
  }

  // Sums of NV doubles per thread over the CTA, in a fixed order, as its
  // partials of slots slot .. slot + NV - 1. (A warp issues one FP64 add per
  // 64 cycles: four warps add three values each, then one warp per sum.)
  template <int NV> __device__ void partial(double (&v)[NV], int slot) {
    const int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < NV; ++j) S.red[j][t] = v[j];
    __syncthreads();
    if (t < 128) {
#pragma unroll
      for (int j = 0; j < NV; ++j)
        S.red[j][t] = (S.red[j][t] + S.red[j][t + 128]) + S.red[j][t + 256];
    }
    __syncthreads();
    if (t < 32 * NV) {
      const double *q = S.red[t >> 5] + lane;
      double x = (q[0] + q[32]) + (q[64] + q[96]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) A.partials[(size_t)(slot + (t >> 5)) * G + bid] = x;
    }
  }

  // A grid barrier, then the totals of slots slot .. slot + N - 1 in a fixed
  // order, the same in every CTA, into tot. A slot is written once an
  // iteration, so no CTA overwrites what another still reads.
  template <int N> __device__ bool totals(int slot) {
    if (!barrier()) return false;
    const int t = threadIdx.x;
    if (t < 32 * N) {
      const double *q = A.partials + (size_t)(slot + (t >> 5)) * G;
      double x = 0.0;
      for (int b = 0; b < G; b += 128) {
        double y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          y[u] = b + 32 * u + lane < G ? __ldcg(q + b + 32 * u + lane) : 0.0;
        x += (y[0] + y[1]) + (y[2] + y[3]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) S.tot[t >> 5] = x;
    }
    __syncthreads();
    return true;
  }

  static __device__ void add(double &d, DF &f, T a, T b) {
    if (sizeof(T) == 8) d = fma((double)a, (double)b, d);
    else df_add_prod(f, (float)a, (float)b);
  }
  static __device__ double total(double d, const DF &f) {
    return sizeof(T) == 8 ? d : df_value(f);
  }

  // Own slices' places in shared memory and their copies.
  __device__ void load() {
    const int t = threadIdx.x;
    if (t < own) {
      const int s = slice(t);
      const int *off = t < tail0 ? A.off2 : A.offA;
      S.rows[t] = A.srows[s];
      S.o[t] = off[s];
      S.w[t] = off[s + 1] - off[s];
    }
    if (t == 0) mbar_init(&S.copies, 1);
    __syncthreads();
    if (t == 0) {
      int used = 0;
      for (int i = 0; i < own; ++i) {
        const int bytes = S.w[i] * (9 * 32 * (int)sizeof(V) + 32 * (int)sizeof(int)) +
                          (uses_d(i) ? 9 * 32 * (int)sizeof(V) : 0);
        S.pos[i] = used + bytes <= A.smem_bytes ? used : -1;
        if (S.pos[i] >= 0) used += bytes;
      }
      mbar_expect_tx(&S.copies, (uint32_t)used);
    }
    __syncthreads();
    if (t < own && S.pos[t] >= 0) {
      const int s = slice(t);
      const size_t o = (size_t)S.o[t];
      unsigned char *dst = mem + S.pos[t];
      const uint32_t vb = (uint32_t)(S.w[t] * 9 * 32 * sizeof(V));
      const uint32_t cb = (uint32_t)(S.w[t] * 32 * sizeof(int));
      if (vb) bulk_g2s(dst, (t < tail0 ? A.val2 : A.valA) + o * 9 * 32, vb, &S.copies);
      if (cb) bulk_g2s(dst + vb, (t < tail0 ? A.col2 : A.colA) + o * 32, cb, &S.copies);
      if (uses_d(t))
        bulk_g2s(dst + vb + cb, A.dmat + (size_t)s * 9 * 32, (uint32_t)(9 * 32 * sizeof(V)),
                 &S.copies);
    }
  }
  // Bounded wait for the copies, by every thread that reads them; a wait
  // that ran out fails the next grid barrier.
  __device__ void wait_copies() {
    unsigned int spins = 0;
    while (!late && !mbar_try_wait(&S.copies, 0)) late = ++spins > kStageSpins;
  }

  static constexpr int kNoLimit = 0x7fffffff;
  template <bool NEG>
  __device__ T row_sum(const V *sv, const int *sc, int w, const T *x, int limit, T a) const {
    return comp_row<V, T, NEG>(sv, sc, w, lane, c, x, limit, a);
  }

  // tail_first (gbilu_reduced.cuh) by component, for own slice i: w is the
  // row's p or s.
  __device__ __forceinline__ void first(int i, bool act, int row, T coef, T w, T *hat) {
    if (slice(i) >= A.S1) return;   // the same for the whole group
    const T a = act ? fma(coef, A.base[3 * row + c], w) : (T)0;
    const T z = comp_d<V, T>(S.xch[grp], grp, c, lane, dblk(i), a);
    if (!act) return;
    const bool split = row - A.n0 < A.split1;
    (split ? A.y : hat)[3 * row + c] = split && !A.transpose ? a : z;
  }

  // The reduced apply's steps after the first sweep of color 1, in step
  // order, a grid barrier around each; w: the row's p or s. A small step's
  // slice belongs to the group that it has in tail(), so a row's own values
  // are this thread's.
  __device__ bool apply(const PhaseList &ph, const T *w, T *hat, T coef) {
    T *y = A.y;
    for (int q = 0; q + 1 < ph.n; ++q) {
      if (!barrier()) return false;
      const Phase &P = ph.p[q];
      const int *off = P.mat ? A.off2 : A.off1r, *col = P.mat ? A.col2 : A.col1r;
      const V *val = P.mat ? A.val2 : A.val1r;
      const int nsl = (P.nrows + 31) >> 5;
      int i0 = (P.slice0 - bid + G - 1) / G;   // the first own slice of the step
      i0 += (grp - (i0 - tail0) % kSmallGroups + kSmallGroups) % kSmallGroups;
      for (int i = i0; slice(i) < P.slice0 + nsl; i += kSmallGroups) {
        const int s = slice(i), r = 32 * (s - P.slice0) + lane, row = P.row0 + r;
        const bool act = r < P.nrows;
        const V *d = A.dmat + (size_t)s * 9 * 32;
        T a = 0;
        if (act) {
          const int e = 3 * row + c;
          const int o = off[s], wd = off[s + 1] - o;
          a = P.own_y ? y[e] : fma(coef, A.base[e], w[e]);
          a = row_sum<true>(val + (size_t)o * 9 * 32, col + (size_t)o * 32, wd,
                                  P.nbr_hat ? hat : y, kNoLimit, a);
        }
        if (P.has_d) a = comp_d<V, T>(S.xch[grp], grp, c, lane, d, a);
        bool fin = true;
        if (P.to_y) {
          fin = row >= P.final0;
          if (act && !fin) y[3 * row + c] = a;
          if (P.final_d) a = comp_d<V, T>(S.xch[grp], grp, c, lane, d, a);
        }
        if (act && fin) hat[3 * row + c] = a;
      }
    }
    if (!barrier()) return false;
    head([&](int i, bool act, int row) {
      T a = 0;
      if (act)
        a = row_sum<true>(vals(i), cols(i), S.w[i], hat, 0x7fffffff,
                                A.base[3 * row + c] * coef);
      if (!A.transpose) a = comp_d<V, T>(S.xch[grp], grp, c, lane, dblk(i), a);
      if (act) hat[3 * row + c] = a;
    });
    return barrier();
  }

  // r0 and the vectors that start from it, ||r0||, base; false: failed run
  __device__ bool start() {
    double d = 0.0, dh = 0.0;
    DF f = {0.f, 0.f}, fh = {0.f, 0.f};
    auto set = [&](int i, int e, T v) {
      A.rt[e] = v;
      if (i < tail0) { A.base[e] = v; add(dh, fh, v, v); }
      else { A.r[e] = v; A.p[e] = v; add(d, f, v, v); }
    };
    if constexpr (sizeof(T) == 8) {
      bool nz = false;
      each(0, own, [&](int i, bool act, int row) {
        if (!act) return;
        const int e = 3 * row + c, g = 3 * A.perm[row] + c;
        const double x = A.from_zero ? 0.0 : A.x_io[g];
        A.x[e] = x;
        A.b[e] = A.b_in[g];
        nz |= x != 0.0;
      });
      if (nz) *A.x_nonzero = 1;
      if (!A.from_zero && !barrier()) return false;
      const bool mul = !A.from_zero && __ldcg(A.x_nonzero) != 0;
      each(0, own, [&](int i, bool act, int row) {
        if (!act) return;
        const int e = 3 * row + c, s = slice(i), o = A.offA[s];
        double q = 0.0;
        if (mul)
          q = row_sum<false>(A.valA + (size_t)o * 9 * 32, A.colA + (size_t)o * 32,
                                    A.offA[s + 1] - o, A.x, kNoLimit, 0.0);
        set(i, e, A.b[e] - q);
      });
    } else {
      each(0, own, [&](int i, bool act, int row) {
        if (!act) return;
        const int e = 3 * row + c;
        A.x[e] = 0;
        set(i, e, (T)(A.scale * A.r64[e]));
      });
    }
    double v[2] = {total(d, f), total(dh, fh)};
    partial(v, 0);
    if (!totals<2>(0)) return false;
    if (threadIdx.x == 0) finish_init<T>(&S.c, S.tot[0] + S.tot[1], 1, S.tot[1]);
    __syncthreads();
    if (S.c.done) return true;
    wait_copies();
    if (A.transpose) {
      head([&](int i, bool act, int row) {
        const T z = comp_d<V, T>(S.xch[grp], grp, c, lane, dblk(i),
                                 act ? A.base[3 * row + c] : (T)0);
        if (act) A.base[3 * row + c] = z;
      });
      if (!barrier()) return false;
    }
    tail([&](int i, bool act, int row) {
      const int e = 3 * row + c, s = slice(i);
      T w = 0;
      if (act) {
        const int o = A.off1[s];
        A.base[e] = row_sum<true>(A.val1 + (size_t)o * 9 * 32, A.col1 + (size_t)o * 32,
                                         A.off1[s + 1] - o, A.base, A.n0, (T)0);
        w = A.p[e];
      }
      first(i, act, row, (T)1, w, A.ph);
    });
    return true;
  }

  __device__ bool iterate(const PhaseList &ph) {
    Ctl &k = S.c;
    while (true) {
      if (!apply(ph, A.p, A.ph, (T)k.cp)) return false;
      {
        double d = 0.0;
        DF f = {0.f, 0.f};
        tail([&](int i, bool act, int row) {
          if (!act) return;
          const int e = 3 * row + c;
          const T a = row_sum<false>(vals(i), cols(i), S.w[i], A.ph, kNoLimit, (T)0);
          A.v[e] = a;
          add(d, f, a, A.rt[e]);
        });
        double v[1] = {total(d, f)};
        partial(v, 2);
        if (!totals<1>(2)) return false;
        if (threadIdx.x == 0) finish_alpha(&k, S.tot[0]);
        __syncthreads();
        if (k.done) return true;
      }
      {
        const T alpha = (T)k.alpha, cs = (T)k.cs;
        double d = 0.0;
        DF f = {0.f, 0.f};
        tail([&](int i, bool act, int row) {
          const int e = 3 * row + c;
          T s = 0;
          if (act) {
            s = fma(-alpha, A.v[e], A.r[e]);
            A.s[e] = s;
            add(d, f, s, s);
          }
          first(i, act, row, cs, s, A.sh);
        });
        if (!apply(ph, A.s, A.sh, cs)) return false;
        double d1 = 0.0, d2 = 0.0;
        DF f1 = {0.f, 0.f}, f2 = {0.f, 0.f};
        tail([&](int i, bool act, int row) {
          if (!act) return;
          const int e = 3 * row + c;
          const T a = row_sum<false>(vals(i), cols(i), S.w[i], A.sh, kNoLimit, (T)0);
          A.t[e] = a;
          add(d1, f1, a, A.s[e]);
          add(d2, f2, a, a);
        });
        double v[3] = {total(d, f), total(d1, f1), total(d2, f2)};
        partial(v, 3);
        if (!totals<3>(3)) return false;
        if (threadIdx.x == 0) {
          finish_s(&k, S.tot[0]);
          if (!k.done) finish_omega(&k, S.tot[1], S.tot[2]);
        }
        __syncthreads();
        if (k.done) return true;
      }
      {
        const T alpha = (T)k.alpha, omega = (T)k.omega;
        double d1 = 0.0, d2 = 0.0;
        DF f1 = {0.f, 0.f}, f2 = {0.f, 0.f};
        tail([&](int i, bool act, int row) {
          if (!act) return;
          const int e = 3 * row + c;
          A.x[e] = fma(omega, A.sh[e], fma(alpha, A.ph[e], A.x[e]));
          const T r = fma(-omega, A.t[e], A.s[e]);
          A.r[e] = r;
          add(d1, f1, r, r);
          add(d2, f2, r, A.rt[e]);
        });
        double v[3] = {total(d1, f1), total(d2, f2), 0.0};
        // the time budget is CTA 0's to judge: one clock for all
        if (A.timeout_ns && bid == 0 && threadIdx.x == 0 &&
            globaltimer() - k.t_start > A.timeout_ns)
          v[2] = 1.0;
        partial(v, 6);
        if (!totals<3>(6)) return false;
        if (threadIdx.x < 32) finish_r(&k, S.tot[0], S.tot[1], S.tot[2] != 0.0);
        __syncthreads();
        if (k.done) return true;
      }
      const T beta = (T)k.beta, omega = (T)k.omega, cp = (T)k.cp;
      const bool restart = k.restart;
      tail([&](int i, bool act, int row) {
        const int e = 3 * row + c;
        T p = 0;
        if (act) {
          const T r = A.r[e];
          p = fma(beta, fma(-omega, A.v[e], A.p[e]), r);
          A.p[e] = p;
          if (restart) A.rt[e] = r;
        }
        first(i, act, row, cp, p, A.ph);
      });
    }
  }

  // x after the loop (k_finish_x, k_finish_head) and the results out
  __device__ bool finish() {
    const Ctl &k = S.c;
    const bool moved = k.half >= 0 && (k.stop_half || k.x_moved);
    if (moved) {
      if (k.stop_half) {
        const T alpha = (T)k.alpha;
        tail([&](int i, bool act, int row) {
          const int e = 3 * row + c;
          if (act) A.x[e] = fma(alpha, A.ph[e], A.x[e]);
        });
      }
      if (!barrier()) return false;
      const T cc = (T)(k.stop_half ? k.cs : k.cr);
      const T *b = sizeof(T) == 8 ? A.b : A.rt;   // the inner solve's b is r0
      head([&](int i, bool act, int row) {
        const int e = 3 * row + c;
        T a = act ? fma(-cc, A.rt[e], b[e]) : (T)0;
        if (A.transpose) a = comp_d<V, T>(S.xch[grp], grp, c, lane, dblk(i), a);
        if (act) a = row_sum<true>(vals(i), cols(i), S.w[i], A.x, kNoLimit, a);
        if (!A.transpose) a = comp_d<V, T>(S.xch[grp], grp, c, lane, dblk(i), a);
        if (act) A.x[e] = a;
      });
    }
    if constexpr (sizeof(T) == 8) {
      if (moved || A.from_zero)
        each(0, own, [&](int i, bool act, int row) {
          if (act) A.x_io[3 * A.perm[row] + c] = A.x[3 * row + c];
        });
    } else {
      // the correction of a run that broke down is dropped
      if (moved && k.status != ST_BREAKDOWN && k.status != ST_NONFINITE)
        each(0, own, [&](int i, bool act, int row) {
          const int e = 3 * row + c;
          if (act) A.x64[e] = fma(A.unscale, (double)A.x[e], A.x64[e]);
        });
    }
    return true;
  }
};

template <typename V, typename T>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_solve_small(const __grid_constant__ SmallArgs<V, T> A, const __grid_constant__ PhaseList ph) {
  extern __shared__ __align__(128) unsigned char small_smem[];
  __shared__ SmallCta<V, T> S;
  SmallSolve<V, T> run(A, S, small_smem);
  if (threadIdx.x == 0) init_ctl(&S.c, A.tol, A.absolute, A.maxit, A.timeout_ns);
  run.load();
  if (run.start() && !S.c.done) run.iterate(ph);
  if (!run.failed) run.finish();
  if (threadIdx.x == 0) run.wait_copies();   // no CTA ends with a copy in flight
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) *A.x_nonzero = 0;
    __syncthreads();
    // the outcome to the host, which sees by host_fail when a wait failed
    const unsigned int *src = reinterpret_cast<const unsigned int *>(&S.c);
    for (int i = threadIdx.x; i < (int)(sizeof(Ctl) / 4); i += kSmallThreads)
      reinterpret_cast<unsigned int *>(A.host_ctl)[i] = src[i];
  }
}

}  // namespace gbilu
