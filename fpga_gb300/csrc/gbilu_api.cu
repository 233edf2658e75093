// C ABI of libgbilu.so (declared in include/gbilu.h): handle lifetime,
// device memory, the BiCGSTAB launch sequence, its CUDA graph (a device-side
// while loop), iterative refinement for the mixed mode and the adjoint.
#include "gbilu.h"
#include "gbilu_fpga_export.hpp"
#include "gbilu_host.hpp"
#include "gbilu_kernels.cuh"
#include "gbilu_reduced.cuh"
#include "gbilu_small.cuh"

#include <algorithm>
#include <chrono>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

namespace gbilu {
namespace {

template <typename T> struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  cudaError_t alloc(size_t count) {
    n = count;
    return cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

// device copy of one sliced matrix
struct DevMat {
  DevBuf<int> off, col;
  DevBuf<int> vsrc;          // source block per slot lane (device factorization)
  bool transpose = false;
  long long slots = 0;
  DevBuf<double> v64;
  DevBuf<float> v32;
  void release() { off.release(); col.release(); vsrc.release(); v64.release(); v32.release(); }
};

// the work vectors of one BiCGSTAB run
template <typename T> struct Vecs {
  DevBuf<T> x, r, rt, p, ph, v, s, sh, t;
  DevBuf<T> y, ysh;          // first sweep of a preconditioner apply (of s)
  DevBuf<T> base;            // reduced iteration (gbilu_reduced.cuh)
  cudaError_t alloc(size_t n) {
    for (DevBuf<T> *b : {&x, &r, &rt, &p, &ph, &v, &s, &sh, &t, &y, &ysh, &base}) {
      cudaError_t e = b->alloc(n);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  void release() {
    for (DevBuf<T> *b : {&x, &r, &rt, &p, &ph, &v, &s, &sh, &t, &y, &ysh, &base}) b->release();
  }
};

// Everything one BiCGSTAB run reads: operator, preconditioner and vectors.
template <typename V, typename T> struct Ops {
  bool transpose;
  const int *offA, *colA; const V *valA;     // A or A^T
  const int *off1, *col1; const V *val1;     // first sweep: L or U^T
  const int *off2, *col2; const V *val2;     // second sweep: U or L^T
  const int *off1r, *col1r; const V *val1r;  // first sweep without color 0's columns
  const V *dmat;                             // Dinv or Dinv^T (sliced)
  Vecs<T> *vec;
};

}  // namespace

constexpr int kMaxChunks = 32;            // of the input values of a factorization

struct Handle {
  gbilu_options opt{};
  std::string err;
  Analysis an;
  bool analyzed = false, factored = false;
  std::vector<double> pvals, lu, dinv;   // host: permuted A, factors
  double analyze_ms = 0, factor_ms = 0, color_ms = 0;
  // device
  bool dev_ready = false;
  int sm_count = 0;
  cudaStream_t st = nullptr, cap = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  // host-buffer solves move b on aux while the initial SpMV runs on st
  // (e_x: x0 is on the device; e_b: b is)
  cudaStream_t aux = nullptr;
  cudaEvent_t e_x = nullptr, e_b = nullptr;
  DevBuf<int2> srows;
  // perm/iperm: device row <-> input row (the vectors of a solve; lambda
  // of the gradient); prowptr, pcol, psrc: the permuted pattern
  DevBuf<int> perm, iperm, prowptr, pcol, psrc;
  DevBuf<int> ibrow, icol;                   // input pattern: block -> row, column (dL/dA)
  DevMat A, L, U, At, Ut, Lt;
  DevMat Lr, Utr;            // L and U^T without color 0's columns
  DevBuf<double> dinv64, dinvT64;
  DevBuf<float> dinv32, dinvT32;
  Vecs<double> v64;
  Vecs<float> v32;
  DevBuf<double> b64, io64, io64b, partials, dA;
  DevBuf<int> x0nz;                        // set when x0 has a nonzero entry
  // device factorization: values in input order (factored in place), inverses
  DevBuf<int> pdiag, bad;
  DevBuf<double> pbuf, vals_in, dinvp;
  // slot lane of each input block in A and in A^T; the input rows by chunk
  // (see plan_chunks), in a chunk by color and input order; input row pointers
  DevBuf<int> apos, tpos, crows, irowptr;
  DevBuf<int> mate, fpos, ftpos, frpos, drow;   // see k_bilu0_rows, FactorOut
  // the input values cross the link in chunks of whole block rows; a color's
  // rows that chunk c completes: run [begin, ready[c]) of each run of colors
  // 0 and 1 (split rows, other rows), see plan_chunks
  struct Run {
    int color, row0, rows;
    std::vector<int> ready;
  };
  std::vector<int> chunk_row, chunk_blk;   // first row, block of each chunk; nb, nnzb
  std::vector<Run> runs;
  cudaEvent_t e_chunk[kMaxChunks] = {};
  bool host_factors_stale = false;
  // color 0's diagonal blocks are well conditioned enough for the reduced
  // iteration (reduced_run)
  bool head_ok = true;
  std::unique_ptr<FpgaExport> fpga;        // the last gbilu_fpga_export (sizes query)
  DevBuf<Ctl> ctl;                         // [0] main run, [1] refinement residual
  Ctl *h_ctl = nullptr;                    // pinned mirror
  bool with_t = false, with_32 = false;
  cudaGraphExec_t graph[2][2][2] = {};     // [reduced][fp32][transpose]
  cudaGraphExec_t graph_ru[2] = {nullptr, nullptr};  // mixed by replacement [transpose]
  int graph_launches[2][2][2] = {}, graph_ru_launches[2] = {};   // kernels an iteration of theirs
  int per_iter[2] = {0, 0};                // launches per iteration [transpose], last run
  long long last_launches = 0;
  // color steps: the full list (one launch per step), and
  // the same as the single-launch apply's parameter when it fits (n = 0
  // otherwise: more than kMaxPhases / 2 colors)
  struct Sweep {
    std::vector<Phase> steps;
    PhaseList phases;
    StagePlan stage = {};                  // shared-memory staging of small steps
    int stage_bytes = 0;
    DevBuf<StageEntry> stage_tab;
    DevBuf<int2> stage_cnt;
    DevBuf<unsigned int> ring_tab;         // streamed slices per CTA (see StagePlan)
    DevBuf<int> ring_cnt;
    void release() {
      stage_tab.release(); stage_cnt.release(); ring_tab.release(); ring_cnt.release();
      stage = StagePlan{};
      stage_bytes = 0;
    }
  };
  Sweep sweep[2][2][2];                    // [reduced][fp32][transpose]
  cudaError_t launch_err = cudaSuccess;    // first failed cooperative launch
  int coop_grid64 = 1, coop_grid32 = 1;    // CTAs of the cooperative apply
  // solves in one launch (gbilu_small.cuh), [fp32]: CTAs (0: not used),
  // dynamic shared memory; their barrier counters, x0 flag and failed wait
  int small_grid[2] = {0, 0}, small_smem[2] = {0, 0};
  DevBuf<unsigned long long> small_bar;
  int *h_fail = nullptr;                   // pinned: a failed wait of one (0: none)
  bool small_probe = false;                // the next one's waits run out (gbilu_wait_probe)
  Ctl *h_inner = nullptr;                  // pinned: an inner solve's outcome
  size_t device_bytes = 0;

  int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    err = buf;
    if (opt.verbose) printf("ERROR: %s\n", buf);
    return code;
  }
};

namespace {

#define CK(call)                                                                 \
  do {                                                                           \
    cudaError_t e_ = (call);                                                     \
    if (e_ != cudaSuccess)                                                       \
      return h->fail(GBILU_CUDA_ERROR, "%s: %s (%s:%d)", #call,                  \
                     cudaGetErrorString(e_), __FILE__, __LINE__);                \
  } while (0)

// the first launch error since the last check (cooperative launches report
// theirs through their return code)
cudaError_t last_error(Handle *h) {
  const cudaError_t e = cudaGetLastError();
  if (h->launch_err != cudaSuccess) {
    const cudaError_t le = h->launch_err;
    h->launch_err = cudaSuccess;
    return le;
  }
  return e;
}

int grid_for(const Handle *h, long long work) {
  long long g = (work + kThreads - 1) / kThreads;
  const long long cap = (long long)h->sm_count * 8;
  return (int)std::max<long long>(1, std::min(g, cap));
}

// Kernels with one thread per entry of a block (kEntryThreads).
int entry_grid(const Handle *h, long long blocks) {
  return (int)std::max<long long>(1, std::min((blocks + 31) / 32, (long long)h->sm_count * 7));
}

// Kernels that end in a grid reduction: fewer, fuller CTAs, so the
// last-CTA step sees few partials and few serialized arrival atomics.
#ifndef GBILU_REDUCE_CTAS_PER_SM
#define GBILU_REDUCE_CTAS_PER_SM 2
#endif
int reduce_grid(const Handle *h, long long work) {
  long long g = (work + kThreads - 1) / kThreads;
  const long long cap = (long long)h->sm_count * GBILU_REDUCE_CTAS_PER_SM;
  return (int)std::max<long long>(1, std::min(g, cap));
}

// k_update_r: 16 bytes a thread and load; CTAs a SM (2: 18.5 us FP64, 12.4 FP32
// for the 500k-cell system's tail, 3: 18.5, 13.6, 4: 21.3, 13.4).
#ifndef GBILU_UPDATE_R_CTAS
#define GBILU_UPDATE_R_CTAS 2
#endif
template <typename T> int update_r_grid(const Handle *h, long long n) {
  const long long g = (n / Pack<T>::N + 2 * kThreads - 1) / (2 * kThreads);
  return (int)std::max<long long>(1, std::min(g, (long long)h->sm_count * GBILU_UPDATE_R_CTAS));
}

// ---------------------------------------------------------------------------
// launch sequences
// ---------------------------------------------------------------------------

// The color steps of one preconditioner apply, in execution order.
// Forward (z = U^-1 L^-1 src): the L sweep over colors 1..C-1 writes y for
// every row (color 0's y is src itself) and the final z = D^-1 y for the
// rows without a higher-colored neighbour; the U sweep then covers color 0
// and the leading rows of colors C-2..1. Transposed (z = L^-T U^-T src): the
// U^T sweep with D^-T over all colors, the rows without a higher-colored
// neighbour final at once (unit diagonal of L^T); the L^T sweep covers the
// leading rows of colors C-2..0.
// reduced: the steps that the reduced iteration leaves to the apply
// (gbilu_reduced.cuh): color 1's first-sweep step is part of the kernel
// before, own values come from base, and color 0 has the last step alone.
std::vector<Phase> make_steps(const Analysis &an, bool transpose, bool reduced = false) {
  std::vector<Phase> st;
  const int C = an.ncolors;
  st.reserve(2 * (size_t)C);
  auto rows = [&](int c) { return an.color_ptr[c + 1] - an.color_ptr[c]; };
  auto add = [&](int c, int mat, int nrows) -> Phase & {
    st.emplace_back();
    Phase &p = st.back();
    p = Phase{};
    p.row0 = an.color_ptr[c];
    p.nrows = nrows;
    p.slice0 = an.slice_color_ptr[c];
    p.mat = mat;
    return p;
  };
  if (reduced) {
    for (int c = 2; c < C; ++c) {
      Phase &p = add(c, 0, rows(c));
      p.has_d = transpose;
      p.own_base = 2;
      p.to_y = 1;
      p.final0 = an.color_ptr[c] + an.split[c];
      p.final_d = !transpose;
    }
    for (int c = C - 2; c >= 0; --c) {
      const int nr = c == 0 ? rows(0) : an.split[c];
      if (nr == 0) continue;
      Phase &p = add(c, 1, nr);
      p.has_d = !transpose;
      p.own_base = c == 0;
      p.own_y = c != 0;
      p.nbr_hat = 1;
    }
  } else if (!transpose) {
    if (C == 1) {   // no couplings: z = D^-1 src
      add(0, 1, rows(0)).has_d = 1;
      return st;
    }
    for (int c = 1; c < C; ++c) {
      Phase &p = add(c, 0, rows(c));
      p.src_rows = an.color_ptr[1];
      p.to_y = 1;
      p.final0 = an.color_ptr[c] + an.split[c];
      p.final_d = 1;
    }
    for (int c = C - 2; c >= 0; --c) {
      const int nr = c == 0 ? rows(0) : an.split[c];
      if (nr == 0) continue;
      Phase &p = add(c, 1, nr);
      p.has_d = 1;
      p.own_y = c == 0 ? 0 : 1;
      p.nbr_hat = 1;
    }
  } else {
    for (int c = 0; c < C; ++c) {
      Phase &p = add(c, 0, rows(c));
      p.has_d = 1;
      p.to_y = 1;
      p.final0 = an.color_ptr[c] + an.split[c];
      p.final_d = 0;
    }
    for (int c = C - 2; c >= 0; --c) {
      if (an.split[c] == 0) continue;
      Phase &p = add(c, 1, an.split[c]);
      p.own_y = 1;
      p.nbr_hat = 1;
    }
  }
  // consecutive single-slice steps (the few rows of the top colors) run on
  // CTA 0, which orders them with a CTA barrier: one grid barrier less each;
  // consecutive small steps, once staged, need no barrier at all: they are
  // ordered by their data (sentinel polling in k_ilu_coop)
  for (size_t q = 0; q + 1 < st.size(); ++q) {
    st[q].local_after = st[q].nrows <= kSliceRows && st[q + 1].nrows <= kSliceRows;
    st[q].flow_after = st[q].nrows <= kSmallRows && st[q + 1].nrows <= kSmallRows;
  }
  return st;
}

// The single-launch apply's parameter (n = 0 when the steps do not fit).
PhaseList phase_list(const std::vector<Phase> &st) {
  PhaseList pl;
  pl.n = 0;
  pl.trace = 0;
  if (st.size() > (size_t)kMaxPhases) return pl;
  for (const Phase &p : st) pl.p[pl.n++] = p;
  return pl;
}

template <typename V, typename T>
int coop_grid(Handle *h) {
  int per_sm = 0, per_sm_red = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ilu_coop<V, T, false>,
                                                coop_threads<T>(), 0);
  if constexpr (sizeof(T) == 4) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_red, k_ilu_coop<V, T, true>,
                                                  coop_threads<T>(), 0);
    per_sm = std::min(per_sm, per_sm_red);
  }
  long long most = 0;
  for (int c = 0; c < h->an.ncolors; ++c) {
    const long long rows = h->an.color_ptr[c + 1] - h->an.color_ptr[c];
    most = std::max(most, rows);
  }
  const int need = (int)((most + coop_threads<T>() - 1) / coop_threads<T>());
  return std::max(1, std::min(per_sm * h->sm_count, need));
}

// Shared-memory staging of the small color steps (see StageEntry): slices are
// dealt round-robin to the CTAs of the cooperative grid; each CTA's entries
// pack [values | column indices | D^-1] at 128-byte multiples. Staging is
// off for this (precision, direction) when a CTA would need more than
// kStageBudget bytes or kMaxStage entries. The large steps' ring takes the
// shared memory left after the staged slices.
constexpr int kStageBudget = 160 * 1024;
// A ring of fewer stages than this leaves compute warps waiting for a
// stage (measured: the FP64 apply, 8 stages of 21.7 KB for 15 compute
// warps, 82 -> 118 us): no ring.
#ifndef GBILU_RING_MIN
#define GBILU_RING_MIN 12
#endif
constexpr int kRingMin = GBILU_RING_MIN;

// Bytes of one slice's [values | column indices | D block] in shared memory.
template <typename V>
long long slice_bytes(const SlicedMatrix &m, int slice, bool uses_d) {
  const long long w = m.off[slice + 1] - m.off[slice];
  return w * 9 * 32 * (long long)sizeof(V) + w * 32 * (long long)sizeof(int) +
         (uses_d ? 9 * 32 * (long long)sizeof(V) : 0);
}

template <typename V, typename T, bool RED>
int build_stage_plan(Handle *h, int f, int t, int grid) {
  Handle::Sweep &sw = h->sweep[RED][f][t];
  PhaseList &pl = sw.phases;
  const Analysis &an = h->an;
  auto mat_of = [&](const Phase &P) -> const SlicedMatrix & {
    if (RED && !P.mat) return t == 0 ? an.Lr : an.Utr;
    return t == 0 ? (P.mat ? an.U : an.L) : (P.mat ? an.Lt : an.Ut);
  };
  std::vector<std::vector<StageEntry>> per(grid);
  std::vector<long long> bytes(grid, 0);
  for (int q = 0; q < pl.n; ++q) {
    Phase &P = pl.p[q];
    P.staged = 0;
    P.streamed = 0;
    if (P.nrows > kSmallRows) continue;
    const SlicedMatrix &m = mat_of(P);
    const int nsl = (P.nrows + kSliceRows - 1) / kSliceRows;
    // steps linked by a CTA barrier (local_after) all run on CTA 0
    const bool local = P.local_after || (q > 0 && pl.p[q - 1].local_after);
    for (int j = 0; j < nsl; ++j) {
      const int b = local ? 0 : (j + q) % grid;
      per[b].push_back(StageEntry{q, j, m.off[P.slice0 + j + 1] - m.off[P.slice0 + j],
                                  (int)bytes[b]});
      bytes[b] += slice_bytes<V>(m, P.slice0 + j, P.uses_d());
    }
    P.staged = 1;
  }
  long long most = 0;
  size_t most_n = 0;
  for (int b = 0; b < grid; ++b) {
    most = std::max(most, bytes[b]);
    most_n = std::max(most_n, per[b].size());
  }
  sw.stage = StagePlan{};
  sw.stage_bytes = 0;
  const bool staged = h->opt.stage_small_steps && most_n > 0 && most <= kStageBudget &&
                      most_n <= (size_t)kMaxStage;
  if (!staged) {
    for (int q = 0; q < pl.n; ++q) pl.p[q].staged = 0;
    most = 0;
  }
  // the ring of the large (not staged) steps, after the staged slices
  int optin = 0;
  CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->opt.device));
  cudaFuncAttributes fa;
  CK(cudaFuncGetAttributes(&fa, k_ilu_coop<V, T, RED>));
  const long long ring_off = (most + 127) / 128 * 128;
  long long stride = 0;
  bool any_large = false;
  // Only a large step that follows another step is streamed: its first
  // stages fill while the steps before it run. The first step of the
  // launch gains nothing from the ring (measured: FP32 L sweep of the
  // 500k-cell system 16.3 us from global memory, 21.2 us streamed).
  auto streamable = [&](int q) {
    const Phase &P = pl.p[q];
    return q > 0 && !P.staged && P.nrows > kSmallRows;
  };
  for (int q = 0; q < pl.n; ++q) {
    const Phase &P = pl.p[q];
    if (!streamable(q)) continue;
    any_large = true;
    const int nsl = (P.nrows + kSliceRows - 1) / kSliceRows;
    for (int j = 0; j < nsl; ++j)
      stride = std::max(stride, slice_bytes<V>(mat_of(P), P.slice0 + j, P.uses_d()));
  }
  stride = (stride + 127) / 128 * 128;
  const long long avail = (long long)optin - (long long)fa.sharedSizeBytes - ring_off;
// Stages of the FP32 ring: 12 is the best of 6..16 on the 500k-cell apply
// (a larger ring leaves less L1 for the large steps that read global
// memory: 8 stages 45.4 us, 12 41.9 us, 16 45.5 us)
#ifndef GBILU_RING_STAGES
#define GBILU_RING_STAGES 12
#endif
  const int ns = (stride > 0 && avail > 0)
                     ? (int)std::min<long long>(GBILU_RING_STAGES, avail / stride) : 0;
  const bool ring = h->opt.stream_large_steps && any_large && ns >= kRingMin;
  if (ring)
    for (int q = 0; q < pl.n; ++q) pl.p[q].streamed = streamable(q);
  const long long dyn = ring ? ring_off + ns * stride : most;
  if (dyn > 0) {
    CK(cudaFuncSetAttribute(k_ilu_coop<V, T, RED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)std::max<long long>(dyn, fa.maxDynamicSharedSizeBytes)));
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ilu_coop<V, T, RED>, coop_threads<T>(),
                                                     (size_t)dyn));
    if (per_sm < 1)
      return h->fail(GBILU_CUDA_ERROR, "single-launch apply does not fit an SM with %lld bytes "
                     "of shared memory", dyn);
  }
  StagePlan sp{nullptr, nullptr, 0, ring ? ns : 0, ring ? (int)stride : 0, (int)ring_off,
               nullptr, nullptr, 0};
  if (ring) {
    // each CTA's streamed slices in launch order: slice j of a step goes to
    // CTA j % grid
    std::vector<std::vector<unsigned int>> lists(grid);
    for (int q = 0; q < pl.n; ++q) {
      const Phase &P = pl.p[q];
      if (!P.streamed) continue;
      const int nsl = (P.nrows + kSliceRows - 1) / kSliceRows;
      for (int j = 0; j < nsl; ++j)
        lists[j % grid].push_back((unsigned int)(P.slice0 + j) | ((unsigned int)P.mat << 30) |
                                  ((unsigned int)P.uses_d() << 31));
    }
    size_t mx = 1;
    for (const auto &l : lists) mx = std::max(mx, l.size());
    std::vector<unsigned int> tab(mx * grid, 0u);
    std::vector<int> cnt(grid);
    for (int b = 0; b < grid; ++b) {
      std::copy(lists[b].begin(), lists[b].end(), tab.begin() + (size_t)b * mx);
      cnt[b] = (int)lists[b].size();
    }
    CK(sw.ring_tab.alloc(tab.size()));
    CK(sw.ring_cnt.alloc(cnt.size()));
    CK(cudaMemcpy(sw.ring_tab.p, tab.data(), tab.size() * sizeof(unsigned int),
                  cudaMemcpyHostToDevice));
    CK(cudaMemcpy(sw.ring_cnt.p, cnt.data(), cnt.size() * sizeof(int), cudaMemcpyHostToDevice));
    sp.ring_tab = sw.ring_tab.p;
    sp.ring_cnt = sw.ring_cnt.p;
    sp.ring_max = (int)mx;
  }
  if (staged) {
    std::vector<StageEntry> tab((size_t)grid * kMaxStage, StageEntry{0, 0, 0, 0});
    std::vector<int2> cnt(grid);
    for (int b = 0; b < grid; ++b) {
      for (size_t e = 0; e < per[b].size(); ++e) tab[(size_t)b * kMaxStage + e] = per[b][e];
      cnt[b] = make_int2((int)per[b].size(), (int)bytes[b]);
    }
    CK(sw.stage_tab.alloc(tab.size()));
    CK(sw.stage_cnt.alloc(cnt.size()));
    CK(cudaMemcpy(sw.stage_tab.p, tab.data(), tab.size() * sizeof(StageEntry),
                  cudaMemcpyHostToDevice));
    CK(cudaMemcpy(sw.stage_cnt.p, cnt.data(), cnt.size() * sizeof(int2),
                  cudaMemcpyHostToDevice));
    sp.tab = sw.stage_tab.p;
    sp.cnt = sw.stage_cnt.p;
    sp.enabled = 1;
  }
  sw.stage = sp;
  sw.stage_bytes = (int)dyn;
  return GBILU_OK;
}

// The single-launch preconditioner apply (cooperative, all CTAs resident).
template <typename V, typename T, bool RED = false>
cudaError_t launch_coop(Handle *h, cudaStream_t s, const Ops<V, T> &o, const T *src, T *hat,
                        int trace, const double *coef = nullptr) {
  const int f = sizeof(T) == 4 ? 1 : 0, t = o.transpose ? 1 : 0;
  const Handle::Sweep &sw = h->sweep[RED][f][t];
  PhaseList pl = sw.phases;
  pl.trace = trace;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(f ? h->coop_grid32 : h->coop_grid64);
  cfg.blockDim = dim3(coop_threads<T>());
  cfg.dynamicSmemBytes = (size_t)sw.stage_bytes;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_ilu_coop<V, T, RED>, h->ctl.p, pl, sw.stage,
                            RED ? o.off1r : o.off1, RED ? o.col1r : o.col1,
                            RED ? o.val1r : o.val1, o.off2, o.col2, o.val2, o.dmat, src,
                            o.vec->y.p, hat, (const T *)o.vec->base.p, coef);
}

// Whether an FP64 apply with two colors is a launch a step. A cooperative launch
// costs more than the launch or two that it saves, but its warps take the
// slices of a step in rounds without a gap between them; it loses again where
// a second round is hardly filled. us in one launch / by steps, by slices of
// the larger color for each of the grid's 2432 warps: 0.03: 24.7 / 16.4, 0.4:
// 26.7 / 22.6, 0.7: 28.7 / 26.7 (a whole gbilu_apply_ilu call 99 / 102), 0.93:
// 28.9 / 30.7, 1.1: 40.6 / 34.9, 1.3: 43.0 / 42.1, 1.44: 43.1 / 42.6 (call 146 /
// 148), 1.56: 43.3 / 46.5, 1.8: 45.2 / 49.4, 2.6: 61.1 / 62.3, 3.9: 80.9 / 84.3,
// 6.4: 130.6 / 129.2, 12.9: 243.9 / 244.1.
bool steps_faster(const Handle *h) {
  const std::vector<int> &c = h->an.slice_color_ptr;
  const double rounds = (double)std::max(c[1], c[2] - c[1]) /
                        (h->sm_count * (coop_threads<double>() / 32));
  return rounds <= 0.6 || (rounds > 1.0 && rounds <= 1.25);
}

// hat = M^-1 src (forward) or M^-T src (transpose); the vector set's y holds
// the first sweep's result. RED: what the reduced iteration leaves of it, with
// coef = &Ctl::cp (src = p) or &Ctl::cs (src = s): in FP32 one launch as well;
// with two colors, or behind k_tail_flow (head_only), the last step alone.
// An FP64 apply with two colors is a launch a step where that is the faster
// form (steps_faster).
template <typename V, typename T, bool RED = false>
void apply_prec(Handle *h, cudaStream_t s, const Ops<V, T> &o, const T *src, T *hat,
                int &launches, const double *coef = nullptr, bool head_only = false) {
  if constexpr (!RED || sizeof(T) == 4) {
    const int C = h->an.ncolors;
    if (h->opt.sweep_mode == 1 && C <= kMaxPhases / 2 &&
        !(C == 2 && (RED || (sizeof(T) == 8 && steps_faster(h))))) {
      const cudaError_t e = launch_coop<V, T, RED>(h, s, o, src, hat, 0, coef);
      if (e != cudaSuccess && h->launch_err == cudaSuccess) h->launch_err = e;
      ++launches;
      return;
    }
  }
  const std::vector<Phase> &steps = h->sweep[RED][sizeof(T) == 4 ? 1 : 0][o.transpose ? 1 : 0].steps;
  for (size_t q = head_only ? steps.size() - 1 : 0; q < steps.size(); ++q) {
    const Phase &P = steps[q];
    k_phase<V, T, RED><<<(unsigned)((P.nrows + kPhaseThreads - 1) / kPhaseThreads), kPhaseThreads, 0, s>>>(
        h->ctl.p, P, P.mat ? o.off2 : RED ? o.off1r : o.off1,
        P.mat ? o.col2 : RED ? o.col1r : o.col1, P.mat ? o.val2 : RED ? o.val1r : o.val1, o.dmat,
        src, o.vec->y.p, hat, o.vec->base.p, coef);
    ++launches;
  }
}

template <typename V, typename T, int MODE>
void spmv(Handle *h, cudaStream_t s, const Ops<V, T> &o, const T *x, T *y, const T *w,
          int &launches, const int *x_nonzero = nullptr, int S0 = 0, Ctl *ctl = nullptr) {
  const int S = h->an.S;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_spmv<V, T, MODE>, kThreads, 0);
  const int grid =
      std::max(1, std::min((S - S0 + kWarps - 1) / kWarps, std::max(1, per_sm) * h->sm_count));
  k_spmv<V, T, MODE><<<grid, kThreads, 0, s>>>(
      ctl ? ctl : h->ctl.p, S0, S, h->srows.p, o.offA, o.colA, o.valA, x, y, w, h->partials.p,
      x_nonzero);
  ++launches;
}

// One full BiCGSTAB iteration (both halves, PROGRAM steps 2-17).
// With ru64 (the FP64 operators; mixed precision by residual replacement)
// the iteration ends with the replacement kernels, which return at once
// unless a replacement is due.
template <typename V, typename T>
void enqueue_iteration(Handle *h, cudaStream_t s, const Ops<V, T> &o,
                       unsigned long long cond, int &launches,
                       const Ops<double, double> *ru64 = nullptr) {
  Vecs<T> &w = *o.vec;
  const int n = 3 * h->an.nb;
  const int g = grid_for(h, n);
  const int gr = reduce_grid(h, n);
  Ctl *c = h->ctl.p;
  double *part = h->partials.p;
  apply_prec(h, s, o, w.p.p, w.ph.p, launches);
  spmv<V, T, SPMV_ALPHA>(h, s, o, w.ph.p, w.v.p, w.rt.p, launches);
  k_update_s<T><<<gr, kThreads, 0, s>>>(c, n, w.r.p, w.v.p, w.s.p, part);
  apply_prec(h, s, o, w.s.p, w.sh.p, launches);
  spmv<V, T, SPMV_OMEGA>(h, s, o, w.sh.p, w.t.p, w.s.p, launches);
  k_update_r<T><<<gr, kThreads, 0, s>>>(c, 0, n, w.x.p, w.ph.p, w.sh.p, w.s.p, w.t.p, w.rt.p,
                                        w.r.p, part, 0, n, w.y.p, w.ysh.p);
  if (ru64 && sizeof(T) == 4) {
    Vecs<double> &d = h->v64;
    k_ru_accumulate<<<g, kThreads, 0, s>>>(c, n, (float *)w.x.p, d.x.p, 0);
    spmv<double, double, SPMV_TRUE>(h, s, *ru64, d.x.p, d.r.p, h->b64.p, launches);
    k_ru_replace<<<gr, kThreads, 0, s>>>(c, n, d.r.p, (float *)w.r.p, (const float *)w.rt.p, part);
    launches += 2;
  }
  k_update_p<T><<<g, kThreads, 0, s>>>(c, n, w.r.p, w.v.p, w.p.p, cond);
  launches += 3;
}

// Whether a run of this handle uses the reduced iteration: not with one color
// (the head would be everything), nor with residual replacement, whose new
// residual is not a multiple of the initial one on the head, nor where color
// 0's diagonal blocks are ill conditioned.
//
// The reduced iteration takes v = p on the head instead of forming A p^ there.
// What it leaves out is the residual of p^ = D^-1 q, about eps |A_00||A_00^-1||q|,
// and it reaches the tail's residual through the multipliers. Scaling rows or
// columns does not matter (both forms change alike; the multipliers' size
// says nothing); the condition of the blocks under the best scaling does, which
// the largest entry of their relative gain arrays measures (Bristol 1966: it is
// the same under any scaling, and 1 for a diagonal block). Attainable residual
// of the reduced form over the full one's (medians of systems of 690 rows
// with blocks multiplied by dense ones, both directions): gain 1: 0.7, 1.6:
// 0.7, 2.6: 0.6-0.95, 4.7: 0.6-1.3, 9: 0.5-2.8, 35: 0.6-16, 2700: 2-2500; rows
// and columns scaled over 1e4 (gain 1.1): 0.6-0.8. Above kMaxHeadGain a run is
// the full iteration.
constexpr double kMaxHeadGain = 4.0;
bool reduced_run(const Handle *h, bool ru) { return h->an.ncolors > 1 && !ru && h->head_ok; }

template <typename V, typename T>
Tail<V, T> make_tail(const Handle *h, const Ops<V, T> &o, T *hat, T *y = nullptr) {
  const Analysis &an = h->an;
  Tail<V, T> P;
  P.row0 = an.color_ptr[1];
  P.rows = an.nb - P.row0;
  P.rows1 = an.color_ptr[2] - P.row0;
  P.split1 = an.split[1];
  P.slice1 = an.slice_color_ptr[1];
  P.d_first = o.transpose;
  P.dmat = o.dmat;
  P.base = o.vec->base.p;
  P.ybuf = y ? y : o.vec->y.p;
  P.hat = hat;
  return P;
}

// CTAs of a kernel with one thread per row.
int row_grid(const Handle *h, int rows, int ctas_per_sm) {
  return std::max(1, std::min((rows + kThreads - 1) / kThreads, h->sm_count * ctas_per_sm));
}

// Whether the small steps run beside the vector kernels (k_tail_flow): FP64,
// three and more colors, few enough for the step list, cooperative launches
// not ruled out by the options, and steps that are small: a few warps of each
// CTA run them with polled loads, a launch of their own costs each about 5 us
// twice an iteration. us an iteration beside / in launches, by rows a step
// (colors, steps):
//   forward 7,800 (10, 16) 522 / 702; 12,900 (6, 8) 201 / 246; 18,800 (6, 8)
//     294 / 305; 23,200 (9, 14) 563 / 586; 28,200 (10, 16) 964 / 945; 38,000
//     (6, 8) 409 / 362
//   adjoint, whose first sweep multiplies by D in every step: 7,800 663 / 706;
//     11,300 (10, 16) 702 / 747; 12,900 238 / 241; 14,400 (8, 12) 521 / 463;
//     18,800 343 / 293; 28,200 1154 / 943; 38,000 467 / 360
// (27-point, nine-point-layer, 30 % fault and random patterns).
constexpr int kFlowRows[2] = {24000, 13000};   // rows a step on average [transpose]
template <typename T> bool flow_run(const Handle *h, bool transpose) {
  const std::vector<Phase> &st = h->sweep[1][0][transpose].steps;
  if (sizeof(T) != 8 || h->an.ncolors < 3 || h->sweep[1][0][transpose].phases.n == 0 ||
      (h->opt.sweep_mode == 0 && !h->opt.one_launch))
    return false;
  long long rows = 0;
  for (size_t q = 0; q + 1 < st.size(); ++q) rows += st[q].nrows;
  return rows <= (long long)kFlowRows[transpose] * (long long)(st.size() - 1);
}

template <int MODE>
void tail_flow(Handle *h, cudaStream_t s, const Ops<double, double> &o, unsigned long long cond,
               int &launches) {
  const PhaseList &pl = h->sweep[1][0][o.transpose].phases;
  Vecs<double> &w = *o.vec;
  long long slices = 0;
  for (int q = 0; q + 1 < pl.n; ++q) slices += (pl.p[q].nrows + kSliceRows - 1) / kSliceRows;
  // one group of three warps for about two slices
  const long long share = 2ll * h->sm_count;
  const Flow F{o.off1r, o.col1r, o.val1r, o.off2, o.col2, o.val2,
               (int)std::max<long long>(1, std::min<long long>(kFlowGroups, (slices + share - 1) / share))};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(h->sm_count);
  cfg.blockDim = dim3(kFlowThreads);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const Tail<double, double> P =
      MODE == 1 ? make_tail(h, o, w.sh.p, w.ysh.p) : make_tail(h, o, w.ph.p, w.y.p);
  const cudaError_t e = cudaLaunchKernelEx(
      &cfg, k_tail_flow<MODE>, h->ctl.p, P, F, pl, (const double *)w.r.p, (const double *)w.v.p,
      MODE == 1 ? w.s.p : w.p.p, w.rt.p, h->partials.p, cond);
  if (e != cudaSuccess && h->launch_err == cudaSuccess) h->launch_err = e;
  ++launches;
}

// One iteration of the reduced form (gbilu_reduced.cuh): the first sweep of
// p on color 1 (and its small steps) was done by the kernel before the loop
// body.
template <typename V, typename T>
void enqueue_reduced(Handle *h, cudaStream_t s, const Ops<V, T> &o, unsigned long long cond,
                     int &launches) {
  Vecs<T> &w = *o.vec;
  Ctl *c = h->ctl.p;
  double *part = h->partials.p;
  const Tail<V, T> tp = make_tail(h, o, w.ph.p), ts = make_tail(h, o, w.sh.p);
  const int S0 = tp.slice1, n0 = 3 * tp.row0, nt = 3 * tp.rows;
  const bool flow = flow_run<T>(h, o.transpose);
  apply_prec<V, T, true>(h, s, o, w.p.p, w.ph.p, launches, &c->cp, flow);
  spmv<V, T, SPMV_ALPHA>(h, s, o, w.ph.p, w.v.p, w.rt.p, launches, nullptr, S0);
  if (flow) {
    if constexpr (sizeof(T) == 8) tail_flow<1>(h, s, o, 0ull, launches);
  } else {
    k_tail_s<V, T><<<row_grid(h, tp.rows, GBILU_REDUCE_CTAS_PER_SM), kThreads, 0, s>>>(
        c, ts, w.r.p, w.v.p, w.s.p, part);
    ++launches;
  }
  apply_prec<V, T, true>(h, s, o, w.s.p, w.sh.p, launches, &c->cs, flow);
  spmv<V, T, SPMV_OMEGA>(h, s, o, w.sh.p, w.t.p, w.s.p, launches, nullptr, S0);
  k_update_r<T><<<update_r_grid<T>(h, nt), kThreads, 0, s>>>(
      c, n0, n0 + nt, w.x.p, w.ph.p, w.sh.p, w.s.p, w.t.p, w.rt.p, w.r.p, part,
      flow ? n0 + 3 * tp.split1 : n0, flow ? n0 + 3 * tp.rows1 : n0 + nt, w.y.p, w.ysh.p);
  ++launches;
  if (flow) {
    if constexpr (sizeof(T) == 8) tail_flow<2>(h, s, o, cond, launches);
  } else {
    k_tail_p<V, T><<<row_grid(h, tp.rows, 8), kThreads, 0, s>>>(c, tp, w.r.p, w.v.p, w.p.p,
                                                                       w.rt.p, cond);
    ++launches;
  }
}

// The reduced form's start, after the initial residual (base holds the
// head's r0): base everywhere and the first sweep of p on color 1.
template <typename V, typename T>
void reduced_start(Handle *h, const Ops<V, T> &o, long long &launches) {
  const Tail<V, T> tp = make_tail(h, o, o.vec->ph.p);
  const bool flow = flow_run<T>(h, o.transpose);
  if (o.transpose) {
    k_base_head<V, T><<<(tp.row0 + kThreads - 1) / kThreads, kThreads, 0, h->st>>>(
        h->ctl.p, tp.row0, o.dmat, o.vec->base.p);
    ++launches;
  }
  const int S = h->an.S;
  k_base_tail<V, T><<<std::min((S - tp.slice1 + kWarps - 1) / kWarps, 8 * h->sm_count), kThreads, 0,
                      h->st>>>(h->ctl.p, tp, S, h->srows.p, o.off1, o.col1, o.val1, o.vec->p.p,
                               o.vec->base.p, flow ? o.vec->sh.p : nullptr, o.vec->ysh.p);
  ++launches;
  if (flow) {
    int l = 0;
    if constexpr (sizeof(T) == 8) tail_flow<0>(h, h->st, o, 0ull, l);
    launches += l;
  }
}

// Blocks up to which a solve (FP64) or an inner solve (FP32) runs in one launch:
// above, a CTA's 12 warps are too few to stream what its shared memory does
// not hold. Later the more steps an apply has: a barrier costs less than a
// launch. us an iteration by the separate kernels / in one launch, by colors
// and 1000 blocks (grids of 7, 9 + 2, 19 and 27 points, faults, random):
//   FP64: 2 colors 742: 86 / 67, 1099: 106 / 98; 3: 1054: 119 / 120; 5: 882: 149 /
//     139, 1069: 159 / 179 (adjoint 179 / 154); 6: 648: 162 / 133, 1082: 201 / 246
//     (238 / 238); 8: 540: 264 / 194, 900: 311 / 325 (397 / 329), 1109: 234 / 270
//     (277 / 259); 10: 1124: 429 / 424, 2146: 522 / 502, 3110: 562 / 579; 10 (banded)
//     1664: 1139 / 834; 15 (random) 1860: 1073 / 1075 (1487 / 1114)
//   FP32: 2 colors 742: 94 / 77, 961: 101 / 96; 3: 676: 93 / 84, 860: 98 / 102; 5: 521:
//     113 / 111, 695: 115 / 122; 6: 648: 180 / 151, 736: 140 / 168, 1082: 165 / 209; 8: 540:
//     266 / 241, 900: 285 / 336, 2208: 217 / 482; 10: 681: 350 / 285, 1124: 347 / 322,
//     1559: 362 / 487; 14: 903: 983 / 1008; 15: 930: 760 / 822
// 170,000 and 140,000 rows are what 7-point grids of those blocks have; with
// fewer blocks a row the vectors decide.
bool one_launch_size(int rows, long long blocks, int colors, bool fp32) {
  if (fp32)
    return rows <= 140000 &&
           blocks <= (colors == 2 ? 970000 : colors > 8 && colors <= 12 ? 1150000 : 700000);
  return rows <= 170000 && blocks <= (colors <= 8 ? 1170000 : 2300000);
}

// Plans the one-launch solve: its CTAs and the shared memory that the
// largest share of slices wants (as much as there is when it is more).
template <typename V, typename T> int plan_small(Handle *h) {
  const Analysis &an = h->an;
  const int f = sizeof(T) == 4;
  h->small_grid[f] = 0;
  if (!h->opt.one_launch || an.ncolors < 2 || !one_launch_size(an.nb, an.nnzb, an.ncolors, f) || h->sweep[1][f][0].phases.n == 0 ||
      h->sweep[1][f][1].phases.n == 0)
    return GBILU_OK;
  const int grid = std::min(h->sm_count, an.S);
  if ((an.S + grid - 1) / grid > kSmallOwn || grid > kSmallThreads) return GBILU_OK;
  cudaFuncAttributes fa;
  int optin = 0;
  CK(cudaFuncGetAttributes(&fa, k_solve_small<V, T>));
  CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->opt.device));
  const int room = optin - (int)fa.sharedSizeBytes;
  std::vector<long long> bytes(grid, 0);
  for (int s = 0; s < an.S; ++s)
    bytes[s % grid] += s < an.slice_color_ptr[1] ? slice_bytes<V>(an.U, s, true)
                                                 : slice_bytes<V>(an.A, s, s < an.slice_color_ptr[2]);
  const int smem = (int)std::min<long long>(room, *std::max_element(bytes.begin(), bytes.end()));
  CK(cudaFuncSetAttribute(k_solve_small<V, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, room));
  int per_sm = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_small<V, T>, kSmallThreads,
                                                   (size_t)smem));
  if (per_sm < 1) return GBILU_OK;
  h->small_grid[f] = grid;
  h->small_smem[f] = smem;
  return GBILU_OK;
}

// The arguments that do not depend on the call.
template <typename V, typename T> SmallArgs<V, T> small_args(Handle *h, const Ops<V, T> &o) {
  const Analysis &an = h->an;
  const int f = sizeof(T) == 4;
  Vecs<T> &w = *o.vec;
  SmallArgs<V, T> A = {};
  A.fail = reinterpret_cast<int *>(h->small_bar.p + 3);
  A.host_fail = h->h_fail;
  A.bar = h->small_bar.p + f;
  A.arrivals = (unsigned int)h->small_grid[f];
  A.spins = kBarrierSpins;
  A.x_nonzero = reinterpret_cast<int *>(h->small_bar.p + 2);
  A.partials = h->partials.p;
  A.srows = h->srows.p;
  A.S = an.S;
  A.S0 = an.slice_color_ptr[1];
  A.S1 = an.slice_color_ptr[2];
  A.n0 = an.color_ptr[1];
  A.split1 = an.split[1];
  A.transpose = o.transpose;
  A.offA = o.offA; A.colA = o.colA; A.valA = o.valA;
  A.off1 = o.off1; A.col1 = o.col1; A.val1 = o.val1;
  A.off1r = o.off1r; A.col1r = o.col1r; A.val1r = o.val1r;
  A.off2 = o.off2; A.col2 = o.col2; A.val2 = o.val2;
  A.dmat = o.dmat;
  A.x = w.x.p; A.r = w.r.p; A.rt = w.rt.p; A.p = w.p.p; A.ph = w.ph.p; A.v = w.v.p;
  A.s = w.s.p; A.sh = w.sh.p; A.t = w.t.p; A.y = w.y.p; A.base = w.base.p;
  A.smem_bytes = h->small_smem[f];
  return A;
}

template <typename V, typename T>
cudaError_t launch_small(Handle *h, SmallArgs<V, T> A) {
  const int f = sizeof(T) == 4;
  *h->h_fail = 0;
  if (h->small_probe) {   // a barrier that one CTA never reaches
    h->small_probe = false;
    A.arrivals += 1;
    A.spins = 1024;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(h->small_grid[f]);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = (size_t)h->small_smem[f];
  cfg.stream = h->st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_solve_small<V, T>, A, h->sweep[1][f][A.transpose].phases);
}

// The outcome of a one-launch solve that has ended, where a wait of it failed:
// its status, and the counters (no longer a multiple of their grid) and the
// mark cleared, in stream order before the next launch.
int check_small(Handle *h, Ctl &c) {
  if (!*h->h_fail) return GBILU_OK;
  c.status = ST_TIMEOUT;
  c.bar_fail = *h->h_fail;
  CK(cudaMemsetAsync(h->small_bar.p, 0, 4 * sizeof(unsigned long long), h->st));
  return GBILU_OK;
}

template <typename V, typename T>
int build_graph(Handle *h, const Ops<V, T> &o, cudaGraphExec_t &exec, int &per_iter,
                const Ops<double, double> *ru64 = nullptr) {
  cudaGraph_t g = nullptr;
  CK(cudaGraphCreate(&g, 0));
  cudaGraphConditionalHandle cond;
  CK(cudaGraphConditionalHandleCreate(&cond, g, 1, cudaGraphCondAssignDefault));
  cudaGraphNodeParams params = {};
  params.type = cudaGraphNodeTypeConditional;
  params.conditional.handle = cond;
  params.conditional.type = cudaGraphCondTypeWhile;
  params.conditional.size = 1;
  cudaGraphNode_t node;
  CK(cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &params));
  cudaGraph_t body = params.conditional.phGraph_out[0];
  CK(cudaStreamBeginCaptureToGraph(h->cap, body, nullptr, nullptr, 0,
                                   cudaStreamCaptureModeThreadLocal));
  int launches = 0;
  if (reduced_run(h, ru64 != nullptr))
    enqueue_reduced(h, h->cap, o, (unsigned long long)cond, launches);
  else
    enqueue_iteration(h, h->cap, o, (unsigned long long)cond, launches, ru64);
  cudaGraph_t captured = nullptr;
  CK(cudaStreamEndCapture(h->cap, &captured));
  CK(cudaGraphInstantiate(&exec, g, 0));
  CK(cudaGraphDestroy(g));
  per_iter = launches;
  return GBILU_OK;
}

template <typename V, typename T> Ops<V, T> make_ops(Handle *h, bool transpose);

template <> Ops<double, double> make_ops(Handle *h, bool t) {
  Ops<double, double> o;
  o.transpose = t;
  DevMat &a = t ? h->At : h->A, &m1 = t ? h->Ut : h->L, &m2 = t ? h->Lt : h->U;
  DevMat &mr = t ? h->Utr : h->Lr;
  o.offA = a.off.p; o.colA = a.col.p; o.valA = a.v64.p;
  o.off1 = m1.off.p; o.col1 = m1.col.p; o.val1 = m1.v64.p;
  o.off2 = m2.off.p; o.col2 = m2.col.p; o.val2 = m2.v64.p;
  o.off1r = mr.off.p; o.col1r = mr.col.p; o.val1r = mr.v64.p;
  o.dmat = t ? h->dinvT64.p : h->dinv64.p;
  o.vec = &h->v64;
  return o;
}

template <> Ops<float, float> make_ops(Handle *h, bool t) {
  Ops<float, float> o;
  o.transpose = t;
  DevMat &a = t ? h->At : h->A, &m1 = t ? h->Ut : h->L, &m2 = t ? h->Lt : h->U;
  DevMat &mr = t ? h->Utr : h->Lr;
  o.offA = a.off.p; o.colA = a.col.p; o.valA = a.v32.p;
  o.off1 = m1.off.p; o.col1 = m1.col.p; o.val1 = m1.v32.p;
  o.off2 = m2.off.p; o.col2 = m2.col.p; o.val2 = m2.v32.p;
  o.off1r = mr.off.p; o.col1r = mr.col.p; o.val1r = mr.v32.p;
  o.dmat = t ? h->dinvT32.p : h->dinv32.p;
  o.vec = &h->v32;
  return o;
}

// Runs the iteration loop of an already initialised Ctl (after the init
// kernels), as a graph or host-driven, then the x fix-up. b: the run's
// right-hand side in the device numbering (only the head's rows are read,
// by the reduced form).
template <typename V, typename T>
int run_loop(Handle *h, bool transpose, int maxit, long long &launches, const T *b, bool ru = false,
             Refine out = {nullptr, 0.0}) {
  Ops<V, T> o = make_ops<V, T>(h, transpose);
  Ops<double, double> o64 = make_ops<double, double>(h, transpose);
  const Ops<double, double> *ru64 = ru ? &o64 : nullptr;
  const int fp32 = sizeof(T) == 4 ? 1 : 0, ti = transpose ? 1 : 0;
  const bool red = reduced_run(h, ru);
  const int n0 = red ? 3 * h->an.color_ptr[1] : 0, n = 3 * h->an.nb - n0;
  if (red) reduced_start(h, o, launches);
  if (h->opt.use_graph) {
    cudaGraphExec_t &gx = ru ? h->graph_ru[ti] : h->graph[red][fp32][ti];
    int &gl = ru ? h->graph_ru_launches[ti] : h->graph_launches[red][fp32][ti];
    if (!gx) {
      int rc = build_graph(h, o, gx, gl, ru64);
      if (rc) return rc;
    }
    h->per_iter[ti] = gl;
    CK(cudaGraphLaunch(gx, h->st));
  } else {
    // host-driven: enqueue two iterations, then look at the done flag
    for (int it = 0; it <= maxit + 1; it += 2) {
      int l = 0;
      for (int k = 0; k < 2; ++k)
        if (red) enqueue_reduced(h, h->st, o, 0ull, l);
        else enqueue_iteration(h, h->st, o, 0ull, l, ru64);
      h->per_iter[ti] = l / 2;
      launches += l;
      CK(cudaMemcpyAsync(h->h_ctl, h->ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
      CK(cudaStreamSynchronize(h->st));
      if (h->h_ctl->done) break;
    }
  }
  k_finish_x<T><<<grid_for(h, n), kThreads, 0, h->st>>>(
      h->ctl.p, n, o.vec->x.p + n0, o.vec->ph.p + n0,
      Refine{out.x64 ? out.x64 + n0 : nullptr, out.scale});
  launches += 1;
  if (red) {
    const int rows = n0 / 3;
    k_finish_head<V, T><<<(rows + kThreads - 1) / kThreads, kThreads, 0, h->st>>>(
        h->ctl.p, rows, transpose, o.off2, o.col2, o.val2, o.dmat, b, o.vec->rt.p, o.vec->x.p,
        out);
    launches += 1;
  }
  CK(last_error(h));
  return GBILU_OK;
}

void fill_result(const Handle *h, const Ctl &c, gbilu_result *res) {
  res->status = c.status;
  res->half_iters = c.status == ST_ALREADY || (c.status == ST_NONFINITE && c.half < 0) ? -1 : c.half;
  res->iterations = res->half_iters / 2.0 + 0.5;
  res->norm0 = c.norm0;
  res->norm = c.norm;
  res->relres = c.norm0 > 0 ? c.norm / c.norm0 : 0.0;
  for (int i = 0; i < 4; ++i) res->norms[i] = c.norms[i];
  res->last_norm_idx = c.last_norm_idx;
  (void)h;
}

// ---------------------------------------------------------------------------
// device set-up
// ---------------------------------------------------------------------------

int upload_mat(Handle *h, const SlicedMatrix &m, DevMat &d) {
  CK(d.off.alloc(m.off.size()));
  CK(d.col.alloc(m.col.size()));
  CK(cudaMemcpy(d.off.p, m.off.data(), m.off.size() * sizeof(int), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(d.col.p, m.col.data(), m.col.size() * sizeof(int), cudaMemcpyHostToDevice));
  const size_t nv = (size_t)m.slots() * 9 * kSliceRows;
  d.slots = m.slots();
  d.transpose = m.transpose_blocks;
  CK(d.v64.alloc(nv));
  if (h->with_32) CK(d.v32.alloc(nv));
  if (h->opt.factor_on_device) {
    CK(d.vsrc.alloc(m.vsrc.size()));
    CK(cudaMemcpy(d.vsrc.p, m.vsrc.data(), m.vsrc.size() * sizeof(int), cudaMemcpyHostToDevice));
    h->device_bytes += m.vsrc.size() * sizeof(int);
  }
  h->device_bytes += (m.off.size() + m.col.size()) * sizeof(int) + nv * 8 + (h->with_32 ? nv * 4 : 0);
  return GBILU_OK;
}

// A sliced value array of the host fill (FP64, entry-major: slots of
// [(slot*9 + e)*32 + l], which is the FP64 device layout) in the device
// layout of V (sl_idx); used for the FP32 copies.
template <typename V>
std::vector<V> to_device_layout(const std::vector<double> &em, size_t slots) {
  std::vector<V> out(em.size());
  for (size_t slot = 0; slot < slots; ++slot)
    for (int e = 0; e < 9; ++e)
      for (int l = 0; l < kSliceRows; ++l)
        out[sl_idx<V>(slot, e, l)] = (V)em[(slot * 9 + e) * kSliceRows + l];
  return out;
}

int upload_vals(Handle *h, const SlicedMatrix &m, const double *src, DevMat &d) {
  const size_t nv = (size_t)m.slots() * 9 * kSliceRows;
  std::vector<double> tmp(nv);
  fill_sliced<double>(m, src, tmp.data());   // the FP64 device layout already
  CK(cudaMemcpy(d.v64.p, tmp.data(), nv * sizeof(double), cudaMemcpyHostToDevice));
  if (h->with_32) {
    const std::vector<float> t32 = to_device_layout<float>(tmp, (size_t)m.slots());
    CK(cudaMemcpy(d.v32.p, t32.data(), nv * sizeof(float), cudaMemcpyHostToDevice));
  }
  return GBILU_OK;
}

int upload_diag(Handle *h, bool transpose, DevBuf<double> &d64, DevBuf<float> &d32) {
  const size_t nv = (size_t)h->an.S * 9 * kSliceRows;
  std::vector<double> tmp(nv);
  fill_sliced_diag<double>(h->an, h->dinv.data(), transpose, tmp.data());
  CK(cudaMemcpy(d64.p, tmp.data(), nv * sizeof(double), cudaMemcpyHostToDevice));
  if (h->with_32) {
    const std::vector<float> t32 = to_device_layout<float>(tmp, (size_t)h->an.S);
    CK(cudaMemcpy(d32.p, t32.data(), nv * sizeof(float), cudaMemcpyHostToDevice));
  }
  return GBILU_OK;
}

void release_device(Handle *h) {
  if (!h->dev_ready) return;
  cudaSetDevice(h->opt.device);
  for (auto &red : h->graph)
    for (auto &row : red)
      for (auto &g : row)
        if (g) { cudaGraphExecDestroy(g); g = nullptr; }
  for (auto &g : h->graph_ru)
    if (g) { cudaGraphExecDestroy(g); g = nullptr; }
  for (DevMat *m : {&h->A, &h->L, &h->U, &h->At, &h->Ut, &h->Lt, &h->Lr, &h->Utr}) m->release();
  for (auto &red : h->sweep)
    for (auto &prec : red)
      for (auto &sw : prec) sw.release();
  h->pdiag.release(); h->bad.release(); h->pbuf.release(); h->vals_in.release();
  h->dinvp.release();
  h->crows.release(); h->irowptr.release(); h->apos.release(); h->tpos.release(); h->mate.release();
  h->fpos.release(); h->ftpos.release(); h->frpos.release(); h->drow.release();
  h->srows.release(); h->perm.release(); h->iperm.release();
  h->ibrow.release(); h->icol.release();
  h->prowptr.release(); h->pcol.release();
  h->psrc.release(); h->dinv64.release(); h->dinvT64.release(); h->dinv32.release();
  h->dinvT32.release(); h->v64.release(); h->v32.release(); h->b64.release();
  h->io64.release(); h->io64b.release(); h->partials.release(); h->dA.release();
  h->x0nz.release();
  h->small_bar.release();
  h->small_grid[0] = h->small_grid[1] = 0;
  h->ctl.release();
  h->device_bytes = 0;
}

// The chunks of a factorization's input and, for each run of rows of colors 0
// and 1 (a color's split rows, its other rows: each in input order), the
// leading rows whose blocks, and whose neighbours', have arrived with chunk
// c. On a grid in natural order that is all but a few layers of the rows up
// to the chunk's end; on any pattern the rows that wait longer are done with
// a later chunk. Returns the input rows by chunk, in a chunk by color.
std::vector<int> plan_chunks(Handle *h) {
  const Analysis &an = h->an;
  // Chunks of 32 MB (160 us on the link; their own kernels take about 100, and
  // launching them delays the next copy's staging by 15), or 8 MB where that
  // gives fewer than six. Factorization of the 500k-cell system with 8, 16,
  // 24, 32, 64 MB and in one piece: 2.06, 1.60, 1.65, 1.57, 1.73, 2.20 ms; of
  // 59,000 cells with 8 MB and in one piece: 0.29, 0.35 ms.
  const long long bytes = (long long)an.nnzb * 72, mb = 1 << 20;
  const int n = (int)std::max<long long>(
      {1, std::min<long long>(bytes / (8 * mb), 6),
       std::min<long long>(bytes / (32 * mb), kMaxChunks)});
  std::vector<int> row_end(n);             // first input row after each chunk
  h->chunk_row.assign(1, 0);
  h->chunk_blk.assign(1, 0);
  for (int c = 0; c < n; ++c) {
    const long long want = (long long)an.nnzb * (c + 1) / n;
    const int row = c + 1 == n ? an.nb
                               : (int)(std::lower_bound(an.rowptr.begin(), an.rowptr.end(), want) -
                                       an.rowptr.begin());
    row_end[c] = std::min(row, an.nb);
    h->chunk_row.push_back(row_end[c]);
    h->chunk_blk.push_back(an.rowptr[row_end[c]]);
  }
  h->runs.clear();
  for (int col = 0; col < std::min(2, an.ncolors); ++col)
    for (int part = 0; part < 2; ++part) {
      const int b = an.color_ptr[col] + (part ? an.split[col] : 0);
      const int e = part ? an.color_ptr[col + 1] : an.color_ptr[col] + an.split[col];
      Handle::Run run{col, b, e - b, std::vector<int>(n, 0)};
      int c = 0;
      for (int i = b; i < e; ++i) {
        const int o = an.perm[i];
        int last = o;
        if (col > 0) last = std::max(o, an.colind[an.rowptr[o + 1] - 1]);
        while (last >= row_end[c]) run.ready[c++] = i - b;   // the prefix so far
      }
      for (; c < n; ++c) run.ready[c] = run.rows;
      h->runs.push_back(std::move(run));
    }
  // a stable pass over the rows in permuted order, color by color
  std::vector<int> chunk_of(an.nb), next(h->chunk_row.begin(), h->chunk_row.end() - 1), rows(an.nb);
  for (int c = 0; c < n; ++c)
    std::fill(chunk_of.begin() + h->chunk_row[c], chunk_of.begin() + h->chunk_row[c + 1], c);
  for (int i = 0; i < an.nb; ++i) rows[next[chunk_of[an.perm[i]]]++] = an.perm[i];
  return rows;
}

// Allocates the device side for the current analysis (structure only).
int setup_device(Handle *h) {
  if (h->opt.device < 0) return h->fail(GBILU_NO_DEVICE, "host-only handle has no device");
  CK(cudaSetDevice(h->opt.device));
  if (!h->st) {
    CK(cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&h->cap, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&h->aux, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&h->e_x, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&h->e_b, cudaEventDisableTiming));
    for (auto &e : h->e_chunk) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    CK(cudaEventCreate(&h->e0));
    CK(cudaEventCreate(&h->e1));
    CK(cudaMallocHost(&h->h_ctl, sizeof(Ctl)));
    CK(cudaMallocHost(&h->h_inner, sizeof(Ctl)));
    CK(cudaMallocHost(&h->h_fail, sizeof(int)));
    CK(cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, h->opt.device));
  }
  release_device(h);
  h->dev_ready = true;
  const Analysis &an = h->an;
  const size_t n = 3 * (size_t)an.nb;
  h->with_t = true;
  h->with_32 = h->opt.precision == GBILU_MIXED;
  std::vector<int2> sr(an.S);
  for (int s = 0; s < an.S; ++s) sr[s] = make_int2(an.slice_row0[s], an.slice_len[s]);
  CK(h->srows.alloc(an.S));
  CK(cudaMemcpy(h->srows.p, sr.data(), sr.size() * sizeof(int2), cudaMemcpyHostToDevice));
  {
    std::vector<int> dv(an.nb), idv(an.nb);
    for (int d = 0; d < an.nb; ++d) {
      dv[d] = an.perm[an.dperm[d]];
      idv[dv[d]] = d;
    }
    CK(h->perm.alloc(an.nb));
    CK(cudaMemcpy(h->perm.p, dv.data(), an.nb * sizeof(int), cudaMemcpyHostToDevice));
    CK(h->iperm.alloc(an.nb));
    CK(cudaMemcpy(h->iperm.p, idv.data(), an.nb * sizeof(int), cudaMemcpyHostToDevice));
  }
  {
    std::vector<int> br(an.nnzb);
    for (int i = 0; i < an.nb; ++i)
      for (int k = an.rowptr[i]; k < an.rowptr[i + 1]; ++k) br[k] = i;
    CK(h->ibrow.alloc(an.nnzb));
    CK(cudaMemcpy(h->ibrow.p, br.data(), an.nnzb * sizeof(int), cudaMemcpyHostToDevice));
    CK(h->icol.alloc(an.nnzb));
    CK(cudaMemcpy(h->icol.p, an.colind.data(), an.nnzb * sizeof(int), cudaMemcpyHostToDevice));
  }
  CK(h->prowptr.alloc(an.nb + 1));
  CK(cudaMemcpy(h->prowptr.p, an.prowptr.data(), (an.nb + 1) * sizeof(int), cudaMemcpyHostToDevice));
  CK(h->pcol.alloc(an.nnzb));
  CK(cudaMemcpy(h->pcol.p, an.pcolind.data(), an.nnzb * sizeof(int), cudaMemcpyHostToDevice));
  CK(h->psrc.alloc(an.nnzb));
  CK(cudaMemcpy(h->psrc.p, an.psrc.data(), an.nnzb * sizeof(int), cudaMemcpyHostToDevice));
  for (auto pr : {std::make_pair(&an.A, &h->A), std::make_pair(&an.L, &h->L),
                  std::make_pair(&an.U, &h->U), std::make_pair(&an.At, &h->At),
                  std::make_pair(&an.Ut, &h->Ut), std::make_pair(&an.Lt, &h->Lt),
                  std::make_pair(&an.Lr, &h->Lr), std::make_pair(&an.Utr, &h->Utr)}) {
    int rc = upload_mat(h, *pr.first, *pr.second);
    if (rc) return rc;
  }
  const size_t nd = (size_t)an.S * 9 * kSliceRows;
  CK(h->dinv64.alloc(nd));
  CK(h->dinvT64.alloc(nd));
  if (h->with_32) { CK(h->dinv32.alloc(nd)); CK(h->dinvT32.alloc(nd)); }
  CK(h->v64.alloc(n));
  if (h->with_32) CK(h->v32.alloc(n));
  CK(h->b64.alloc(n));
  CK(h->io64.alloc(n));
  CK(h->io64b.alloc(n));
  const size_t maxgrid = std::max<size_t>((size_t)h->sm_count * 8, (size_t)(an.S + kWarps - 1) / kWarps) + 1;
  CK(h->partials.alloc(2 * maxgrid));
  CK(h->x0nz.alloc(1));
  CK(cudaMemset(h->x0nz.p, 0xff, sizeof(int)));   // "nonzero" until a gather clears it
  CK(h->ctl.alloc(2));
  CK(cudaMemset(h->ctl.p, 0, 2 * sizeof(Ctl)));
  CK(h->small_bar.alloc(4));
  CK(cudaMemset(h->small_bar.p, 0, 4 * sizeof(unsigned long long)));
  if (h->opt.factor_on_device) {
    CK(h->pdiag.alloc(an.nb));
    CK(cudaMemcpy(h->pdiag.p, an.pdiag.data(), an.nb * sizeof(int), cudaMemcpyHostToDevice));
    CK(h->bad.alloc(2));
    CK(h->pbuf.alloc((size_t)an.nnzb * 9));
    CK(h->vals_in.alloc((size_t)an.nnzb * 9));
    CK(h->dinvp.alloc((size_t)an.nb * 9));
    // the sliced arrays are written block by block: their padding stays zero
    for (DevMat *m : {&h->A, &h->At, &h->L, &h->U, &h->Lt, &h->Ut, &h->Lr, &h->Utr}) {
      CK(cudaMemsetAsync(m->v64.p, 0, m->v64.n * sizeof(double), h->st));
      if (h->with_32) CK(cudaMemsetAsync(m->v32.p, 0, m->v32.n * sizeof(float), h->st));
    }
    CK(cudaMemsetAsync(h->dinv64.p, 0, nd * sizeof(double), h->st));
    CK(cudaMemsetAsync(h->dinvT64.p, 0, nd * sizeof(double), h->st));
    if (h->with_32) {
      CK(cudaMemsetAsync(h->dinv32.p, 0, nd * sizeof(float), h->st));
      CK(cudaMemsetAsync(h->dinvT32.p, 0, nd * sizeof(float), h->st));
    }
    // where each block goes: apos, tpos by input block, the others by permuted
    // block (of a diagonal block: unused)
    for (DevBuf<int> *b : {&h->apos, &h->tpos, &h->mate, &h->fpos, &h->ftpos, &h->frpos})
      CK(b->alloc(an.nnzb));
    CK(cudaMemsetAsync(h->frpos.p, 0xff, an.nnzb * sizeof(int), h->st));
    CK(h->drow.alloc(an.nb));
    CK(cudaMemcpyAsync(h->drow.p, an.idperm.data(), an.nb * sizeof(int), cudaMemcpyHostToDevice, h->st));
    const int gi = grid_for(h, an.nnzb);
    k_mates<<<grid_for(h, an.nb), kThreads, 0, h->st>>>(an.nb, h->prowptr.p, h->pcol.p, h->pdiag.p,
                                                        h->psrc.p, h->mate.p);
    auto positions = [&](DevMat &m, const int *psrc, DevBuf<int> &pos) {
      if (m.slots)
        k_block_positions<<<gi, kThreads, 0, h->st>>>(m.slots * 32, m.vsrc.p, psrc, pos.p);
      h->device_bytes -= (size_t)m.slots * 32 * sizeof(int);
    };
    positions(h->A, h->psrc.p, h->apos);
    positions(h->At, h->psrc.p, h->tpos);
    positions(h->L, nullptr, h->fpos);
    positions(h->U, nullptr, h->fpos);
    positions(h->Lt, nullptr, h->ftpos);
    positions(h->Ut, nullptr, h->ftpos);
    positions(h->Lr, nullptr, h->frpos);
    positions(h->Utr, nullptr, h->frpos);
    CK(cudaStreamSynchronize(h->st));
    CK(cudaGetLastError());
    for (DevMat *m : {&h->A, &h->At, &h->L, &h->U, &h->Lt, &h->Ut, &h->Lr, &h->Utr})
      m->vsrc.release();
    const std::vector<int> crows = plan_chunks(h);
    CK(h->crows.alloc(an.nb));
    CK(cudaMemcpy(h->crows.p, crows.data(), an.nb * sizeof(int), cudaMemcpyHostToDevice));
    CK(h->irowptr.alloc(an.nb + 1));
    CK(cudaMemcpy(h->irowptr.p, an.rowptr.data(), (an.nb + 1) * sizeof(int), cudaMemcpyHostToDevice));
    h->device_bytes += (size_t)an.nnzb * 24 + (size_t)an.nb * 12;
    h->device_bytes += (size_t)an.nnzb * 9 * 16 + (size_t)an.nb * 76;
  }
  for (int red = 0; red < 2; ++red)
    for (int f = 0; f < 2; ++f)
      for (int t = 0; t < 2; ++t) {
        Handle::Sweep &sw = h->sweep[red][f][t];
        if (red && an.ncolors == 1) sw.steps.clear();
        else sw.steps = make_steps(an, t != 0, red != 0);
        sw.phases = phase_list(sw.steps);
      }
  h->coop_grid64 = coop_grid<double, double>(h);
  h->coop_grid32 = coop_grid<float, float>(h);
  if (an.ncolors <= kMaxPhases / 2) {
    for (int t = 0; t < 2; ++t) {
      int rc = build_stage_plan<double, double, false>(h, 0, t, h->coop_grid64);
      if (rc) return rc;
      if (h->with_32) {
        rc = build_stage_plan<float, float, false>(h, 1, t, h->coop_grid32);
        if (rc) return rc;
        rc = build_stage_plan<float, float, true>(h, 1, t, h->coop_grid32);
        if (rc) return rc;
      }
    }
  }
  if (h->with_32) {
    if (h->opt.mixed_scheme == 0)
      if (int rc = plan_small<float, float>(h)) return rc;
  } else if (int rc = plan_small<double, double>(h)) {
    return rc;
  }
  h->device_bytes += nd * 16 + (h->with_32 ? nd * 8 : 0) + n * 8 * 15 + (h->with_32 ? n * 4 * 12 : 0) +
                     (size_t)an.nnzb * 16 + (size_t)an.nb * 16;
  return GBILU_OK;
}

FactorOut factor_out(Handle *h) {
  return FactorOut{h->fpos.p, h->ftpos.p, h->frpos.p, h->drow.p,
                   h->L.v64.p, h->U.v64.p, h->Lt.v64.p, h->Ut.v64.p, h->Lr.v64.p, h->Utr.v64.p,
                   h->dinv64.p, h->dinvT64.p,
                   h->L.v32.p, h->U.v32.p, h->Lt.v32.p, h->Ut.v32.p, h->Lr.v32.p, h->Utr.v32.p,
                   h->dinv32.p, h->dinvT32.p};
}

// Factors rows row_a .. and row_b .. of one color.
void bilu0_rows(Handle *h, const FactorOut &F, int color, int row_a, int rows_a, int row_b = 0,
                int rows_b = 0) {
  const int rows = rows_a + rows_b;
  if (rows <= 0) return;
  k_bilu0_rows<<<(rows + kBiluRows - 1) / kBiluRows, kThreads, 0, h->st>>>(
      row_a, rows_a, row_b, rows_b, h->an.color_ptr[color], h->an.slice_color_ptr[color],
      h->prowptr.p, h->pcol.p, h->pdiag.p, h->psrc.p, h->mate.p, h->pbuf.p,
      h->dinvp.p, F, h->bad.p);
}

// Permute, factor and lay out on the device: the values (host array, input
// order) cross the link in chunks on the auxiliary stream; behind each, its
// rows go into A and A^T, and the rows of colors 0 and 1 that it completes are
// factored, into L, U, U^T, L^T and the inverse
// diagonal blocks; then the other colors. 500k cells: 2.81 -> 1.57 ms, of
// which the link alone takes 1.1.
int factor_device(Handle *h, const double *vals) {
  const Analysis &an = h->an;
  CK(cudaMemsetAsync(h->bad.p, 0x7f, 2 * sizeof(int), h->st));
  const int none = 0x7f7f7f7f;
  // the values of an earlier factorization may still be read on st
  CK(cudaEventRecord(h->e_x, h->st));
  CK(cudaStreamWaitEvent(h->aux, h->e_x, 0));
  const FactorOut F = factor_out(h);
  const int n = (int)h->chunk_row.size() - 1;
  for (int c = 0; c < n; ++c) {
    const int r0 = h->chunk_row[c], nr = h->chunk_row[c + 1] - r0;
    const size_t v0 = 9 * (size_t)h->chunk_blk[c];
    const size_t bytes = (9 * (size_t)h->chunk_blk[c + 1] - v0) * sizeof(double);
    if (nr > 0) {
      CK(cudaMemcpyAsync(h->vals_in.p + v0, vals + v0, bytes, cudaMemcpyHostToDevice, h->aux));
      CK(cudaEventRecord(h->e_chunk[c], h->aux));
      CK(cudaStreamWaitEvent(h->st, h->e_chunk[c], 0));
      CK(cudaMemcpyAsync(h->pbuf.p + v0, h->vals_in.p + v0, bytes, cudaMemcpyDeviceToDevice, h->st));
      k_scatter_rows<<<std::min((nr + 31) / 32, 8 * h->sm_count), kThreads, 0, h->st>>>(
          nr, h->crows.p + r0, h->irowptr.p, h->vals_in.p, h->apos.p, h->tpos.p, h->A.v64.p,
          h->At.v64.p, h->with_32 ? h->A.v32.p : nullptr, h->with_32 ? h->At.v32.p : nullptr);
    }
    for (size_t q = 0; q + 1 < h->runs.size(); q += 2) {   // a color's two runs
      const Handle::Run &a = h->runs[q], &b = h->runs[q + 1];
      const int fa = c ? a.ready[c - 1] : 0, fb = c ? b.ready[c - 1] : 0;
      bilu0_rows(h, F, a.color, a.row0 + fa, a.ready[c] - fa, b.row0 + fb, b.ready[c] - fb);
    }
  }
  for (int c = 2; c < an.ncolors; ++c)
    bilu0_rows(h, F, c, an.color_ptr[c], an.color_ptr[c + 1] - an.color_ptr[c]);
  int *bad = reinterpret_cast<int *>(h->h_inner);   // pinned
  CK(cudaMemcpyAsync(bad, h->bad.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  if (*bad != none)
    return h->fail(GBILU_SINGULAR,
                   "gbilu_factor: singular diagonal block in permuted row %d (input row %d)", *bad,
                   an.perm[*bad]);
  // compared by its high word, that of a gain below the limit is below the limit's
  const uint64_t limit = (uint64_t)(uint32_t)-bad[1] << 32;
  double gain;
  memcpy(&gain, &limit, sizeof gain);
  h->head_ok = gain < kMaxHeadGain;
  h->host_factors_stale = true;
  return GBILU_OK;
}

int check_solve_ready(Handle *h) {
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  if (!h->factored) return h->fail(GBILU_NOT_READY, "gbilu_factor has not been called");
  if (h->opt.device < 0) return h->fail(GBILU_NO_DEVICE, "host-only handle cannot solve");
  return GBILU_OK;
}

// FP64 BiCGSTAB on the permuted vectors: b in h->b64, x in v64.x.
// With sync false the final Ctl is only queued for copy into h->h_ctl: the
// caller synchronizes once at the end (no host round trip mid-solve).
// b_ready: an event after which b is on the device (it is moved on another
// stream while A x0 is computed), or null when it is ready in stream order.
// b_in: b in the input numbering (permuted as it is read), or null for b64.
int solve64(Handle *h, bool transpose, double tol, int maxit, Ctl &out, long long &launches,
            bool sync = true, cudaEvent_t b_ready = nullptr, const double *b_in = nullptr) {
  const int n = 3 * h->an.nb;
  Ops<double, double> o = make_ops<double, double>(h, transpose);
  Vecs<double> &w = h->v64;
  const unsigned long long tmo = (unsigned long long)(h->opt.timeout_ms * 1e6);
  k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, tol, h->opt.absolute_tol, maxit, tmo);
  int l = 1;
  // r = A x0 (zeros without reading A when the gather of x0 found none)
  spmv<double, double, SPMV_PLAIN>(h, h->st, o, w.x.p, w.r.p, nullptr, l, h->x0nz.p);
  launches += l;
  if (b_ready) CK(cudaStreamWaitEvent(h->st, b_ready, 0));
  const int nh = reduced_run(h, false) ? 3 * h->an.color_ptr[1] : 0;
  k_init_resid<double><<<reduce_grid(h, n), kThreads, 0, h->st>>>(
      h->ctl.p, n, nh, b_in ? b_in : h->b64.p, b_in ? h->perm.p : nullptr, h->b64.p, w.r.p, w.rt.p,
      w.p.p, w.base.p, h->partials.p);
  launches += 1;
  int rc = run_loop<double, double>(h, transpose, maxit, launches, h->b64.p);
  if (rc) return rc;
  CK(cudaMemcpyAsync(h->h_ctl, h->ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
  if (!sync) return GBILU_OK;
  CK(cudaStreamSynchronize(h->st));
  out = *h->h_ctl;
  if (h->opt.use_graph) launches += (long long)out.body_runs * h->per_iter[transpose ? 1 : 0];
  return GBILU_OK;
}

// Mixed precision by residual replacement: FP32 storage, sweeps and
// vectors, the FP32 correction accumulated into the FP64 x and the FP32
// residual replaced by the FP64 b - A x whenever the recursive residual fell
// by ru_delta (and when it reaches the bound); the stop is decided on the
// FP64 residual. The Krylov space is never restarted. b in h->b64, x in
// v64.x (FP64, permuted).
int solve_mixed_ru(Handle *h, bool transpose, double tol, int maxit, gbilu_result *res,
                   Ctl &out, long long &launches) {
  const int n = 3 * h->an.nb;
  Ops<double, double> o64 = make_ops<double, double>(h, transpose);
  Vecs<double> &w = h->v64;
  Vecs<float> &f = h->v32;
  const unsigned long long tmo = (unsigned long long)(h->opt.timeout_ms * 1e6);
  k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, tol, h->opt.absolute_tol, maxit, tmo);
  int l = 0;
  spmv<double, double, SPMV_RESID>(h, h->st, o64, w.x.p, w.r.p, h->b64.p, l);
  k_ru_init<<<reduce_grid(h, n), kThreads, 0, h->st>>>(h->ctl.p, n, h->opt.ru_delta, w.r.p, f.r.p,
                                                       f.rt.p, f.p.p, f.x.p, h->partials.p);
  launches += l + 2;
  int rc = run_loop<float, float>(h, transpose, maxit, launches, nullptr, true);
  if (rc) return rc;
  // a stop after a first half owes xc += alpha p^ (k_finish_x in run_loop);
  // then the remaining FP32 correction goes into x
  k_ru_accumulate<<<grid_for(h, n), kThreads, 0, h->st>>>(h->ctl.p, n, f.x.p, w.x.p, 1);
  launches += 1;
  CK(cudaMemcpyAsync(h->h_ctl, h->ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  out = *h->h_ctl;
  if (h->opt.use_graph) launches += (long long)out.body_runs * h->per_iter[transpose ? 1 : 0];
  if (out.status == ST_ALREADY || (out.status == ST_NONFINITE && out.half < 0)) return GBILU_OK;
  // report the FP64 residual of the returned x (recomputed unless the last
  // replacement just did)
  double tn = out.true_norm;
  if (out.status != ST_OK) {
    Ctl *outer = h->ctl.p + 1;
    k_ctl_init<<<1, 32, 0, h->st>>>(outer, 0.0, 1, 0, 0ull);
    l = 1;
    spmv<double, double, SPMV_RESID>(h, h->st, o64, w.x.p, w.r.p, h->b64.p, l, nullptr, 0, outer);
    launches += l;
    CK(cudaMemcpyAsync(h->h_ctl, outer, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    tn = h->h_ctl->norm0;
  }
  out.norm = tn;
  if (res) {
    res->outer_iters = out.replacements;
    res->inner_half_iters = out.half + 1;
    res->true_relres = out.norm0 > 0 ? tn / out.norm0 : 0.0;
  }
  return GBILU_OK;
}

// Mixed precision: FP32 inner BiCGSTAB inside FP64 iterative refinement.
// b in h->b64, x in v64.x (FP64, permuted).
int solve_mixed(Handle *h, bool transpose, double tol, int maxit, gbilu_result *res,
                Ctl &out, long long &launches) {
  if (h->opt.mixed_scheme == 1) return solve_mixed_ru(h, transpose, tol, maxit, res, out, launches);
  const int n = 3 * h->an.nb;
  Ops<double, double> o64 = make_ops<double, double>(h, transpose);
  Vecs<double> &w = h->v64;
  Vecs<float> &f = h->v32;
  Ctl *outer = h->ctl.p + 1;
  auto enqueue_residual = [&]() -> int {
    // r = b - A x in FP64 with the FP64 copy of A, ||r|| into h_ctl
    k_ctl_init<<<1, 32, 0, h->st>>>(outer, 0.0, 1, 0, 0ull);
    int l = 1;
    spmv<double, double, SPMV_RESID>(h, h->st, o64, w.x.p, w.r.p, h->b64.p, l, nullptr, 0, outer);
    launches += l;
    CK(cudaMemcpyAsync(h->h_ctl, outer, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
    return GBILU_OK;
  };
  int rc = enqueue_residual();
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->st));
  const double nrm0 = h->h_ctl->norm0;
  double nrm = nrm0;
  memset(&out, 0, sizeof out);
  out.norm0 = nrm0;
  out.norms[0] = nrm0;
  out.status = ST_MAXIT;
  if (!std::isfinite(nrm0)) { out.status = ST_NONFINITE; out.half = -1; out.norm = nrm0; return GBILU_OK; }
  const double bound = h->opt.absolute_tol ? tol : tol * nrm0;
  if (!(nrm0 > (h->opt.absolute_tol ? tol : kAlreadySolved))) {
    out.status = ST_ALREADY; out.half = -1; out.norm = nrm0;
    return GBILU_OK;
  }
  const unsigned long long tmo = (unsigned long long)(h->opt.timeout_ms * 1e6);
  int outer_steps = 0, inner_half = 0;
  // maxit caps the inner half-iterations of all refinement steps together
  // the way the reference caps one run: at most maxit full iterations plus
  // the first half of one more, 2*maxit + 1 halves (solver.vhd:557). Each
  // inner solve gets the full iterations that still fit.
  const long long budget = 2LL * maxit + 1;
  const bool small = h->small_grid[1] > 0 && reduced_run(h, false);
  if (small) h->per_iter[transpose ? 1 : 0] = 0;
  while (nrm > bound && outer_steps < h->opt.max_outer && inner_half < budget) {
    const int left = (int)std::min<long long>((budget - inner_half - 1) / 2, h->opt.inner_maxit);
    // the correction A d = r / ||r|| in FP32 from d = 0, x += ||r|| d unless it
    // broke down, the next residual behind it, and one look at both
    if (small) {   // all but the residual in one launch
      SmallArgs<float, float> A = small_args(h, make_ops<float, float>(h, transpose));
      A.host_ctl = h->h_inner;
      A.r64 = w.r.p;
      A.x64 = w.x.p;
      A.scale = 1.0 / nrm;
      A.unscale = nrm;
      A.tol = h->opt.inner_tol;
      A.maxit = left;
      A.timeout_ns = tmo;
      CK(launch_small(h, A));
      ++launches;
    } else {
      k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, h->opt.inner_tol, 0, left, tmo);
      const int nh = reduced_run(h, false) ? 3 * h->an.color_ptr[1] : 0;
      k_init_rhs<<<reduce_grid(h, n), kThreads, 0, h->st>>>(h->ctl.p, n, nh, 1.0 / nrm, w.r.p,
                                                            f.r.p, f.rt.p, f.p.p, f.x.p, f.base.p,
                                                            h->partials.p);
      // the inner run starts from x = 0: its right-hand side is rt
      rc = run_loop<float, float>(h, transpose, left, launches, f.rt.p, false, Refine{w.x.p, nrm});
      if (rc) return rc;
      launches += 2;
      CK(cudaMemcpyAsync(h->h_inner, h->ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
    }
    rc = enqueue_residual();
    if (rc) return rc;
    CK(cudaStreamSynchronize(h->st));
    CK(last_error(h));
    Ctl ic = *h->h_inner;
    if (small) rc = check_small(h, ic);
    else if (h->opt.use_graph) launches += (long long)ic.body_runs * h->per_iter[transpose ? 1 : 0];
    if (rc) return rc;
    inner_half += (ic.half >= 0 ? ic.half + 1 : 0);
    ++outer_steps;
    if (ic.status == ST_BREAKDOWN || ic.status == ST_NONFINITE) { out.status = ic.status; break; }
    nrm = h->h_ctl->norm0;
    if (!std::isfinite(nrm)) { out.status = ST_NONFINITE; break; }
    if (ic.status == ST_TIMEOUT) { out.status = ST_TIMEOUT; break; }
  }
  if (nrm <= bound) out.status = ST_OK;
  out.norm = nrm;
  // the counter of one run that did all inner halves back to back
  out.half = inner_half - 1;
  if (res) {
    res->outer_iters = outer_steps;
    res->inner_half_iters = inner_half;
    res->true_relres = nrm0 > 0 ? nrm / nrm0 : 0.0;
  }
  out.norms[1] = nrm;
  out.last_norm_idx = 1;
  return GBILU_OK;
}

}  // namespace
}  // namespace gbilu

namespace gbilu {
namespace {
// Algorithmic bytes of one iteration's kernels as they run (every operand
// read or written once, x gathers counted once).
struct IterBytes {
  double apply, spmv, update_s, update_r, update_p;
  double total() const { return 2 * apply + 2 * spmv + update_s + update_r + update_p; }
};
IterBytes iter_bytes(const Handle *h, double sv, double sx) {
  const Analysis &an = h->an;
  const double si = 4.0, blk = 9 * sv + si, nb = an.nb, row = 3 * sx;
  IterBytes b;
  if (!reduced_run(h, false)) {
    b.apply = ((double)an.nnzb_l + an.nnzb_u) * blk + 2 * (nb + 1) * si + nb * 9 * sv + 4 * nb * row;
    b.spmv = an.nnzb * blk + (nb + 1) * si + 3 * nb * row;
    b.update_s = 3 * nb * row;
    b.update_r = 8 * nb * row;
    b.update_p = 4 * nb * row;
    return b;
  }
  const double n0 = an.color_ptr[1], nt = nb - n0, n1 = an.color_ptr[2] - n0, split = an.split[1];
  const double a0 = an.prowptr[an.color_ptr[1]], u0 = a0 - n0;   // the head's blocks of A and U
  // apply: the head's U blocks and D; base and result of the head, the tail's
  // result gathered
  b.apply = u0 * blk + n0 * 9 * sv + (n0 + 1) * si + (2 * n0 + nt) * row;
  b.spmv = (an.nnzb - a0) * blk + (nt + 1) * si + (nb + 2 * nt) * row;
  const double d1 = (n1 - split) * 9 * sv;
  b.update_s = 5 * nt * row + d1;    // r, v, base -> s, s^ of color 1
  b.update_r = 8 * nt * row;
  b.update_p = 6 * nt * row + d1;    // r, v, p, base -> p, p^ of color 1
  // the small steps, in the apply or beside the vector kernels: the L and U
  // blocks inside the tail, D of its rows but color 1's final ones
  const double small = ((double)an.nnzb_l + an.nnzb_u - 2 * u0) * blk + (nt - n1 + split) * 9 * sv;
  if (sv == 8 && flow_run<double>(h, false)) {
    b.update_s += small;
    b.update_p += small;
  } else {
    b.apply += small;
  }
  return b;
}

// One of the iteration's kernels for gbilu_bench_kernel (kind 3: the
// iteration's apply, 4: SpMV with the alpha dot, 5: SpMV with the omega dots,
// 6-8: update_s/r/p), over the rows that it runs on.
template <typename V, typename T>
void iter_kernel(Handle *h, int kind, const Ops<V, T> &o, int n, int g, int gr, int &l) {
  Vecs<T> &w = *o.vec;
  if (reduced_run(h, false)) {
    const Tail<V, T> tp = make_tail(h, o, w.ph.p), ts = make_tail(h, o, w.sh.p);
    const int S0 = tp.slice1, n0 = 3 * tp.row0, nt = 3 * tp.rows;
    Ctl *c = h->ctl.p;
    const bool flow = flow_run<T>(h, o.transpose);
    if (kind == 3) {
      apply_prec<V, T, true>(h, h->st, o, w.p.p, w.ph.p, l, &c->cp, flow);
      return;
    }
    if (flow && kind == 6) {
      if constexpr (sizeof(T) == 8) tail_flow<1>(h, h->st, o, 0ull, l);
      return;
    }
    if (flow && kind == 8) {
      if constexpr (sizeof(T) == 8) tail_flow<2>(h, h->st, o, 0ull, l);
      return;
    }
    if (kind == 4) {
      spmv<V, T, SPMV_ALPHA>(h, h->st, o, w.ph.p, w.v.p, w.rt.p, l, nullptr, S0);
      return;
    }
    if (kind == 5) {
      spmv<V, T, SPMV_OMEGA>(h, h->st, o, w.ph.p, w.t.p, w.s.p, l, nullptr, S0);
      return;
    }
    if (kind == 6)
      k_tail_s<V, T><<<row_grid(h, tp.rows, GBILU_REDUCE_CTAS_PER_SM), kThreads, 0, h->st>>>(
          c, ts, w.r.p, w.v.p, w.s.p, h->partials.p);
    else if (kind == 7)
      k_update_r<T><<<update_r_grid<T>(h, nt), kThreads, 0, h->st>>>(
          c, n0, n0 + nt, w.x.p, w.ph.p, w.sh.p, w.s.p, w.t.p, w.rt.p, w.r.p, h->partials.p,
          flow ? n0 + 3 * tp.split1 : n0, flow ? n0 + 3 * tp.rows1 : n0 + nt, w.y.p, w.ysh.p);
    else
      k_tail_p<V, T><<<row_grid(h, tp.rows, 8), kThreads, 0, h->st>>>(c, tp, w.r.p, w.v.p, w.p.p,
                                                                       w.rt.p, 0ull);
    ++l;
    return;
  }
  if (kind == 3) {
    apply_prec<V, T>(h, h->st, o, w.p.p, w.ph.p, l);
  } else if (kind == 4) {
    spmv<V, T, SPMV_ALPHA>(h, h->st, o, w.p.p, w.v.p, w.rt.p, l);
  } else if (kind == 5) {
    spmv<V, T, SPMV_OMEGA>(h, h->st, o, w.p.p, w.t.p, w.s.p, l);
  } else if (kind == 6) {
    k_update_s<T><<<gr, kThreads, 0, h->st>>>(h->ctl.p, n, w.r.p, w.v.p, w.s.p, h->partials.p);
    ++l;
  } else if (kind == 7) {
    k_update_r<T><<<gr, kThreads, 0, h->st>>>(h->ctl.p, 0, n, w.x.p, w.ph.p, w.sh.p, w.s.p, w.t.p,
                                              w.rt.p, w.r.p, h->partials.p, 0, n, w.y.p, w.ysh.p);
    ++l;
  } else {
    k_update_p<T><<<g, kThreads, 0, h->st>>>(h->ctl.p, n, w.r.p, w.v.p, w.p.p, 0ull);
    ++l;
  }
}
}  // namespace
}  // namespace gbilu

using namespace gbilu;

extern "C" {

int gbilu_default_options(gbilu_options *o) {
  if (!o) return GBILU_BAD_INPUT;
  memset(o, 0, sizeof *o);
  o->precision = GBILU_FP64;
  o->absolute_tol = 0;
  o->device = 0;
  o->use_graph = 1;
  o->timeout_ms = 0.0;
  o->inner_tol = 1e-1;
  o->inner_maxit = 500;
  o->max_outer = 30;
  o->verbose = 0;
  o->sweep_mode = 1;
  o->factor_on_device = 0;
  o->mixed_scheme = 0;
  o->ru_delta = 0.1;
  o->stage_small_steps = 1;
  o->coloring = 0;
  o->stream_large_steps = 0;
  o->color_on_device = 0;
  o->one_launch = 1;
  return GBILU_OK;
}

int gbilu_create(const gbilu_options *opt, void **handle) {
  if (!handle) return GBILU_BAD_INPUT;
  *handle = nullptr;
  Handle *h = new (std::nothrow) Handle();
  if (!h) return GBILU_BAD_INPUT;
  if (opt) h->opt = *opt; else gbilu_default_options(&h->opt);
  if (h->opt.precision != GBILU_FP64 && h->opt.precision != GBILU_MIXED) {
    delete h;
    return GBILU_BAD_INPUT;
  }
  *handle = h;
  return GBILU_OK;
}

int gbilu_destroy(void *handle) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (h->st) {
    cudaSetDevice(h->opt.device);
    cudaStreamSynchronize(h->st);
    release_device(h);
    cudaStreamDestroy(h->st);
    cudaStreamDestroy(h->cap);
    cudaStreamDestroy(h->aux);
    cudaEventDestroy(h->e_x);
    cudaEventDestroy(h->e_b);
    for (auto &e : h->e_chunk) cudaEventDestroy(e);
    cudaEventDestroy(h->e0);
    cudaEventDestroy(h->e1);
    cudaFreeHost(h->h_ctl);
    cudaFreeHost(h->h_inner);
    cudaFreeHost(h->h_fail);
  }
  delete h;
  return GBILU_OK;
}

int gbilu_analyze(void *handle, int nb, const int *rowptr, const int *colind) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  auto t0 = std::chrono::steady_clock::now();
  h->analyzed = h->factored = false;
  h->head_ok = true;
  h->fpga.reset();
  if (h->opt.coloring != 0 && h->opt.coloring != 1)
    return h->fail(GBILU_BAD_INPUT, "gbilu_analyze: coloring must be 0 or 1");
  std::vector<int> dcolors;
  h->color_ms = 0.0;
  if (h->opt.color_on_device && h->opt.device >= 0 && h->opt.coloring == 0) {
    // the pattern is checked first: the device coloring assumes it is valid
    std::string perr = check_pattern(nb, rowptr, colind);
    if (!perr.empty()) return h->fail(GBILU_BAD_INPUT, "gbilu_analyze: %s", perr.c_str());
    dcolors.resize(nb);
    int nc = 0;
    perr = color_parity_device(nb, rowptr, colind, h->opt.device, dcolors.data(), &nc, &h->color_ms);
    if (!perr.empty())
      return h->fail(GBILU_CUDA_ERROR, "gbilu_analyze: device coloring: %s", perr.c_str());
  }
  std::string err = analyze(nb, rowptr, colind, h->an, true, h->opt.coloring,
                            dcolors.empty() ? nullptr : dcolors.data(),
                            dcolors.empty() ? &h->color_ms : nullptr);
  if (!err.empty()) return h->fail(GBILU_BAD_INPUT, "gbilu_analyze: %s", err.c_str());
  h->analyzed = true;
  if (h->opt.device >= 0) {
    int rc = setup_device(h);
    if (rc) return rc;
  }
  h->analyze_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  if (h->opt.verbose)
    printf("INFO: gbilu_analyze: nb=%d nnzb=%d colors=%d slices=%d (%.1f ms)\n", nb, h->an.nnzb,
           h->an.ncolors, h->an.S, h->analyze_ms);
  return GBILU_OK;
}

int gbilu_get_ordering(void *handle, int *ncolors, int *color, int *perm, int *color_ptr) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  if (ncolors) *ncolors = h->an.ncolors;
  if (color) memcpy(color, h->an.color.data(), h->an.nb * sizeof(int));
  if (perm) memcpy(perm, h->an.perm.data(), h->an.nb * sizeof(int));
  if (color_ptr) memcpy(color_ptr, h->an.color_ptr.data(), (h->an.ncolors + 1) * sizeof(int));
  return GBILU_OK;
}

int gbilu_factor(void *handle, const double *vals) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  if (!vals) return h->fail(GBILU_BAD_INPUT, "vals must not be NULL");
  auto t0 = std::chrono::steady_clock::now();
  h->factored = false;
  h->fpga.reset();
  const Analysis &an = h->an;
  if (h->opt.factor_on_device && h->opt.device >= 0) {
    CK(cudaSetDevice(h->opt.device));
    h->pvals.clear();   // the host copies are only made when asked for
    const int rc = factor_device(h, vals);
    if (rc) return rc;
    h->factored = true;
    h->factor_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return GBILU_OK;
  }
  h->host_factors_stale = false;
  h->pvals.resize((size_t)an.nnzb * 9);
  permute_values(an, vals, h->pvals.data());
  h->lu = h->pvals;
  h->dinv.assign((size_t)an.nb * 9, 0.0);
  const int bad = bilu0(an, h->lu.data(), h->dinv.data());
  if (bad >= 0)
    return h->fail(GBILU_SINGULAR, "gbilu_factor: singular diagonal block in permuted row %d (input row %d)",
                   bad, an.perm[bad]);
  h->head_ok = head_gain(an, h->lu.data(), h->dinv.data()) < kMaxHeadGain;
  if (h->opt.device >= 0) {
    CK(cudaSetDevice(h->opt.device));
    int rc;
    if ((rc = upload_vals(h, an.A, h->pvals.data(), h->A))) return rc;
    if ((rc = upload_vals(h, an.L, h->lu.data(), h->L))) return rc;
    if ((rc = upload_vals(h, an.U, h->lu.data(), h->U))) return rc;
    if ((rc = upload_vals(h, an.At, h->pvals.data(), h->At))) return rc;
    if ((rc = upload_vals(h, an.Ut, h->lu.data(), h->Ut))) return rc;
    if ((rc = upload_vals(h, an.Lt, h->lu.data(), h->Lt))) return rc;
    if ((rc = upload_vals(h, an.Lr, h->lu.data(), h->Lr))) return rc;
    if ((rc = upload_vals(h, an.Utr, h->lu.data(), h->Utr))) return rc;
    if ((rc = upload_diag(h, false, h->dinv64, h->dinv32))) return rc;
    if ((rc = upload_diag(h, true, h->dinvT64, h->dinvT32))) return rc;
  }
  h->factored = true;
  h->factor_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return GBILU_OK;
}

int gbilu_get_factors(void *handle, double *lu, double *dinv) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!h->factored) return h->fail(GBILU_NOT_READY, "gbilu_factor has not been called");
  if (h->host_factors_stale) {      // factored on the device: fetch the copies
    CK(cudaSetDevice(h->opt.device));
    h->lu.resize((size_t)h->an.nnzb * 9);
    h->dinv.resize((size_t)h->an.nb * 9);
    std::vector<double> in(h->lu.size());   // input order -> permuted order
    CK(cudaMemcpy(in.data(), h->pbuf.p, in.size() * sizeof(double), cudaMemcpyDeviceToHost));
    permute_values(h->an, in.data(), h->lu.data());
    CK(cudaMemcpy(h->dinv.data(), h->dinvp.p, h->dinv.size() * sizeof(double),
                  cudaMemcpyDeviceToHost));
    h->host_factors_stale = false;
  }
  if (lu) memcpy(lu, h->lu.data(), h->lu.size() * sizeof(double));
  if (dinv) memcpy(dinv, h->dinv.data(), h->dinv.size() * sizeof(double));
  return GBILU_OK;
}

int gbilu_fpga_export(void *handle, const double *b, const double *x0, int *vector_sizes,
                      int *nnz_sizes, void *const *vp) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!h->factored) return h->fail(GBILU_NOT_READY, "gbilu_factor has not been called");
  int rc = gbilu_get_factors(h, nullptr, nullptr);   // host copies of the factors
  if (rc) return rc;
  const Analysis &an = h->an;
  if (h->pvals.size() != (size_t)an.nnzb * 9) {
    // factored on the device: the permuted A from the uploaded input values
    std::vector<double> in((size_t)an.nnzb * 9);
    CK(cudaSetDevice(h->opt.device));
    CK(cudaMemcpy(in.data(), h->vals_in.p, in.size() * sizeof(double), cudaMemcpyDeviceToHost));
    h->pvals.resize(in.size());
    permute_values(an, in.data(), h->pvals.data());
  }
  if (!vp || !h->fpga) {
    auto ex = std::make_unique<FpgaExport>();
    const std::string err = fpga_export(an, h->pvals.data(), h->lu.data(), h->dinv.data(), *ex);
    if (!err.empty()) return h->fail(GBILU_BAD_INPUT, "gbilu_fpga_export: %s", err.c_str());
    h->fpga = std::move(ex);
  }
  const FpgaExport &ex = *h->fpga;
  if (vector_sizes) memcpy(vector_sizes, ex.vector_sizes, sizeof ex.vector_sizes);
  if (nnz_sizes) memcpy(nnz_sizes, ex.nnz_sizes, sizeof ex.nnz_sizes);
  if (!vp) return GBILU_OK;
  for (int m = 0; m < 3; ++m) {
    void *const *v = vp + 6 * m;
    if (!v[0] || !v[1] || !v[2] || !*(double *const *)v[2] || !v[3] || !v[4])
      return h->fail(GBILU_BAD_INPUT, "gbilu_fpga_export: a vector pointer is NULL");
    memcpy(v[0], ex.sizes[m].data(), ex.sizes[m].size() * sizeof(unsigned int));
    memcpy(v[1], ex.pidx[m].data(), ex.pidx[m].size() * sizeof(unsigned int));
    memcpy(*(double *const *)v[2], ex.vals[m].data(), ex.vals[m].size() * sizeof(double));
    memcpy(v[3], ex.cols[m].data(), ex.cols[m].size() * sizeof(unsigned short));
    memcpy(v[4], ex.nrs[m].data(), ex.nrs[m].size());
  }
  if (!vp[18] || !vp[19] || !vp[20])
    return h->fail(GBILU_BAD_INPUT, "gbilu_fpga_export: a vector pointer is NULL");
  memcpy(vp[18], ex.blkdiag.data(), ex.blkdiag.size() * sizeof(double));
  // rhs and x0 in the permuted numbering of the exported rows
  double *rhs = static_cast<double *>(vp[19]), *xx = static_cast<double *>(vp[20]);
  for (int i = 0; i < an.nb; ++i)
    for (int r = 0; r < 3; ++r) {
      rhs[3 * i + r] = b ? b[3 * (size_t)an.perm[i] + r] : 0.0;
      xx[3 * i + r] = x0 ? x0[3 * (size_t)an.perm[i] + r] : 0.0;
    }
  return GBILU_OK;
}

// One solve through the ABI. With gx and gdA (the adjoint), after the
// transposed solve the gradient dL/dA = -lambda_i x_j^T is formed on the
// device from lambda (still in the device vector) and gx (the forward
// solution, input numbering), inside the timed region, into gdA (input
// block order; host or device like the other arrays).
// from_zero: x0 = 0, and x is only written.
static int solve_impl(Handle *h, const double *b, double *x, bool device_ptrs, bool transpose,
                      double tol, int maxit, gbilu_result *res, const double *gx = nullptr,
                      double *gdA = nullptr, bool from_zero = false) {
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (!b || !x) return h->fail(GBILU_BAD_INPUT, "b and x must not be NULL");
  if (maxit < 0) return h->fail(GBILU_BAD_INPUT, "maxit must be >= 0");
  if (!(tol >= 0.0)) return h->fail(GBILU_BAD_INPUT, "tol must be >= 0");
  auto t0 = std::chrono::steady_clock::now();
  CK(cudaSetDevice(h->opt.device));
  const int nb = h->an.nb, n = 3 * nb;
  const int g = grid_for(h, n);
  long long launches = 0;
  Ctl c;
  gbilu_result tmp;
  memset(&tmp, 0, sizeof tmp);
  gbilu_result *r = res ? res : &tmp;
  memset(r, 0, sizeof *r);
  const bool fp64 = h->opt.precision != GBILU_MIXED;
  const bool small = fp64 && h->small_grid[0] > 0 && reduced_run(h, false);
  if (small) h->per_iter[transpose ? 1 : 0] = 0;
  CK(cudaEventRecord(h->e0, h->st));
  // One launch reads b and x0 and writes x in the caller's numbering; host
  // arrays go through staging copies.
  if (small) {
    const double *db = b;
    double *dx = x;
    if (!device_ptrs) {
      if (!from_zero)
        CK(cudaMemcpyAsync(h->io64b.p, x, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
      CK(cudaMemcpyAsync(h->io64.p, b, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
      db = h->io64.p;
      dx = h->io64b.p;
    }
    // dL/dA reads gx after this launch wrote lambda: where the caller's two
    // arrays overlap, lambda stays in the staging buffer until then
    const bool overlap = device_ptrs && gx && gdA && (uintptr_t)x < (uintptr_t)(gx + n) &&
                         (uintptr_t)gx < (uintptr_t)(x + n);
    if (overlap) dx = h->io64b.p;
    SmallArgs<double, double> A = small_args(h, make_ops<double, double>(h, transpose));
    A.host_ctl = h->h_ctl;
    A.b = h->b64.p;
    A.perm = h->perm.p;
    A.b_in = db;
    A.x_io = dx;
    A.from_zero = from_zero;
    A.tol = tol;
    A.absolute = h->opt.absolute_tol;
    A.maxit = maxit;
    A.timeout_ns = (unsigned long long)(h->opt.timeout_ms * 1e6);
    CK(launch_small(h, A));
    ++launches;
    if (gx && gdA) {   // lambda is in the input numbering already
      const double *xin = gx;
      if (!device_ptrs) {   // b's staging buffer is free once the solve read it
        CK(cudaMemcpyAsync(h->io64.p, gx, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
        xin = h->io64.p;
      }
      k_grad_a<<<entry_grid(h, h->an.nnzb), kEntryThreads, 0, h->st>>>(
          h->an.nnzb, h->ibrow.p, h->icol.p, dx, xin, device_ptrs ? gdA : h->dA.p);
      ++launches;
      if (overlap)
        CK(cudaMemcpyAsync(x, dx, n * sizeof(double), cudaMemcpyDeviceToDevice, h->st));
    }
    CK(cudaEventRecord(h->e1, h->st));
    if (!device_ptrs)
      CK(cudaMemcpyAsync(x, dx, n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  }
  if (!small) {
    const double *db = b;
    const double *dx = x;
    double *mapped_x = nullptr;
    if (!device_ptrs) {
      // Page-locked host buffers are read and written by the gather/scatter
      // kernels in place (mapped, over the CPU-GPU link); other host memory
      // goes through staging copies.
      cudaPointerAttributes ab, ax;
      const bool zb = cudaPointerGetAttributes(&ab, b) == cudaSuccess &&
                      ab.type == cudaMemoryTypeHost && ab.devicePointer;
      const bool zx = cudaPointerGetAttributes(&ax, x) == cudaSuccess &&
                      ax.type == cudaMemoryTypeHost && ax.devicePointer;
      cudaGetLastError();   // a query on unregistered memory is not an error here
      if (zb && zx) {
        db = static_cast<const double *>(ab.devicePointer);
        dx = mapped_x = static_cast<double *>(ax.devicePointer);
      } else {
        db = h->io64.p;   // staging copies below
        dx = h->io64b.p;
      }
    }
    // The FP64 solve needs b only after A x0 (k_init_resid): from host
    // buffers, b moves on the auxiliary stream while the SpMV runs. The
    // CPU-GPU link is one shared budget (about 200 GB/s for reads and writes
    // together, measured), so x0 goes first and alone; b follows on the copy
    // engine, which takes no SMs from the SpMV, and is permuted on the device.
    const bool overlap_b = fp64 && !device_ptrs;
    if (!device_ptrs && !mapped_x && !from_zero)
      CK(cudaMemcpyAsync(h->io64b.p, x, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
    CK(cudaMemsetAsync(h->x0nz.p, 0, sizeof(int), h->st));
    if (from_zero)
      CK(cudaMemsetAsync(h->v64.x.p, 0, n * sizeof(double), h->st));
    else if (mapped_x)   // host side read in order, device side written permuted
      k_scatter<double><<<g, kThreads, 0, h->st>>>(nb, h->iperm.p, dx, h->v64.x.p, h->x0nz.p);
    else
      k_gather<double, double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, dx, h->v64.x.p, 1.0,
                                                          h->x0nz.p);
    cudaStream_t sb = h->st;
    if (overlap_b) {
      CK(cudaEventRecord(h->e_x, h->st));
      CK(cudaStreamWaitEvent(h->aux, h->e_x, 0));
      sb = h->aux;
    }
    if (!device_ptrs && (!mapped_x || overlap_b)) {
      CK(cudaMemcpyAsync(h->io64.p, b, n * sizeof(double), cudaMemcpyHostToDevice, sb));
      db = h->io64.p;
    }
    if (overlap_b)   // k_init_resid permutes b as it reads it
      CK(cudaEventRecord(h->e_b, h->aux));
    else if (mapped_x)
      k_scatter<double><<<g, kThreads, 0, sb>>>(nb, h->iperm.p, db, h->b64.p);
    else
      k_gather<double, double><<<g, kThreads, 0, sb>>>(nb, h->perm.p, db, h->b64.p, 1.0);
    launches += overlap_b ? 1 : 2;
    if (!fp64)
      rc = solve_mixed(h, transpose, tol, maxit, r, c, launches);
    else
      rc = solve64(h, transpose, tol, maxit, c, launches, false, overlap_b ? h->e_b : nullptr,
                   overlap_b ? db : nullptr);
    if (rc) return rc;
    if (gx && gdA) {
      // lambda from the device numbering into the input numbering (x comes
      // in it), then dL/dA in the input block order
      const double *xin = gx;
      if (!device_ptrs) {   // b's staging buffer is free once the solve read it
        CK(cudaMemcpyAsync(h->io64.p, gx, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
        xin = h->io64.p;
      }
      k_scatter<double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, h->v64.x.p, h->v64.r.p);
      k_grad_a<<<entry_grid(h, h->an.nnzb), kEntryThreads, 0, h->st>>>(
          h->an.nnzb, h->ibrow.p, h->icol.p, h->v64.r.p, xin, device_ptrs ? gdA : h->dA.p);
      launches += 2;
    }
    // x back to the caller's numbering. When the initial residual already met
    // the bound, v64.x still holds x0 (gathered), so this returns x0 unchanged
    // bit for bit; the FP64 path therefore needs no status before it and the
    // whole solve ends in one host synchronization.
    if (mapped_x)   // device side read permuted, host side written in order
      k_gather<double, double><<<g, kThreads, 0, h->st>>>(nb, h->iperm.p, h->v64.x.p, mapped_x, 1.0);
    else
      k_scatter<double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, h->v64.x.p,
                                                   device_ptrs ? x : h->io64b.p);
    launches += 1;
    CK(cudaEventRecord(h->e1, h->st));
    if (!device_ptrs && !mapped_x)
      CK(cudaMemcpyAsync(x, h->io64b.p, n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  }
  if (gx && gdA && !device_ptrs)
    CK(cudaMemcpyAsync(gdA, h->dA.p, (size_t)h->an.nnzb * 9 * sizeof(double),
                       cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  if (fp64) {
    c = *h->h_ctl;
    if (h->opt.use_graph) launches += (long long)c.body_runs * h->per_iter[transpose ? 1 : 0];
    if (small) {
      rc = check_small(h, c);
      if (rc) return rc;
      // after a failed wait x has not been written: zero where it was to be
      // (as by a run that ends before its first iteration), and dL/dA with it
      if (c.bar_fail && from_zero) {
        const size_t xb = n * sizeof(double);
        const size_t ab = gx && gdA ? (size_t)h->an.nnzb * 9 * sizeof(double) : 0;
        if (device_ptrs) {
          CK(cudaMemsetAsync(x, 0, xb, h->st));
          if (ab) CK(cudaMemsetAsync(gdA, 0, ab, h->st));
          CK(cudaStreamSynchronize(h->st));
        } else {
          memset(x, 0, xb);
          if (ab) memset(gdA, 0, ab);
        }
      }
    }
  }
  const int outer = r->outer_iters, inner = r->inner_half_iters;
  const double tr = r->true_relres;
  fill_result(h, c, r);
  r->outer_iters = outer;
  r->inner_half_iters = inner;
  r->true_relres = h->opt.precision == GBILU_MIXED ? tr : r->relres;
  float ms = 0;
  CK(cudaEventElapsedTime(&ms, h->e0, h->e1));
  r->device_ms = ms;
  r->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  h->last_launches = launches;
  if (h->opt.verbose)
    printf("INFO: gbilu_solve: status=%d half_iters=%d relres=%.3e device %.3f ms\n", r->status,
           r->half_iters, r->relres, r->device_ms);
  return GBILU_OK;
}

int gbilu_solve(void *handle, const double *b, double *x, double tol, int maxit, gbilu_result *res) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  return solve_impl(h, b, x, false, false, tol, maxit, res);
}

int gbilu_solve_from_zero(void *handle, const double *b, double *x, double tol, int maxit,
                          gbilu_result *res) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  return solve_impl(h, b, x, false, false, tol, maxit, res, nullptr, nullptr, true);
}

int gbilu_solve_device(void *handle, const double *d_b, double *d_x, double tol, int maxit,
                       gbilu_result *res) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  return solve_impl(h, d_b, d_x, true, false, tol, maxit, res);
}

int gbilu_apply_spmv(void *handle, const double *x, double *y, int transpose) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (!x || !y) return h->fail(GBILU_BAD_INPUT, "x and y must not be NULL");
  CK(cudaSetDevice(h->opt.device));
  const int nb = h->an.nb, n = 3 * nb, g = grid_for(h, n);
  Ops<double, double> o = make_ops<double, double>(h, transpose != 0);
  Vecs<double> &w = h->v64;
  int launches = 0;
  CK(cudaMemcpyAsync(h->io64.p, x, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
  k_gather<double, double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, h->io64.p, w.p.p, 1.0);
  spmv<double, double, SPMV_PLAIN>(h, h->st, o, w.p.p, w.v.p, nullptr, launches);
  k_scatter<double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, w.v.p, h->io64b.p);
  CK(cudaMemcpyAsync(y, h->io64b.p, n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  h->last_launches = launches + 2;
  return GBILU_OK;
}

int gbilu_apply_ilu(void *handle, const double *p, double *z, int transpose) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (!p || !z) return h->fail(GBILU_BAD_INPUT, "p and z must not be NULL");
  CK(cudaSetDevice(h->opt.device));
  const int nb = h->an.nb, n = 3 * nb, g = grid_for(h, n);
  const bool t = transpose != 0;
  Ops<double, double> o = make_ops<double, double>(h, t);
  Vecs<double> &w = h->v64;
  int launches = 0;
  k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, 0.0, 0, 0, 0ull);
  CK(cudaMemcpyAsync(h->io64.p, p, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
  k_gather<double, double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, h->io64.p, w.p.p, 1.0);
  apply_prec(h, h->st, o, w.p.p, w.ph.p, launches);
  k_scatter<double><<<g, kThreads, 0, h->st>>>(nb, h->perm.p, w.ph.p, h->io64b.p);
  CK(cudaMemcpyAsync(z, h->io64b.p, n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  h->last_launches = launches + 3;
  return GBILU_OK;
}

int gbilu_adjoint(void *handle, const double *g_in, const double *x, double *lambda, double *dA,
                  double tol, int maxit, gbilu_result *res) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!g_in || !x || !lambda) return h->fail(GBILU_BAD_INPUT, "g, x and lambda must not be NULL");
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (dA && h->dA.n != (size_t)h->an.nnzb * 9) {
    CK(cudaSetDevice(h->opt.device));
    h->dA.release();
    CK(h->dA.alloc((size_t)h->an.nnzb * 9));
  }
  // lambda = A^-T g: the transposed solve, x0 = 0, then dL/dA on the device
  return solve_impl(h, g_in, lambda, false, true, tol, maxit, res, dA ? x : nullptr, dA, true);
}

int gbilu_adjoint_device(void *handle, const double *d_g, const double *d_x, double *d_lambda,
                         double *d_dA, double tol, int maxit, gbilu_result *res) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!d_g || !d_x || !d_lambda)
    return h->fail(GBILU_BAD_INPUT, "g, x and lambda must not be NULL");
  int rc = check_solve_ready(h);
  if (rc) return rc;
  return solve_impl(h, d_g, d_lambda, true, true, tol, maxit, res, d_dA ? d_x : nullptr, d_dA,
                    true);
}

int gbilu_get_stats(void *handle, gbilu_stats *s) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h || !s) return GBILU_BAD_INPUT;
  memset(s, 0, sizeof *s);
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  const Analysis &an = h->an;
  s->nb = an.nb;
  s->nnzb = an.nnzb;
  s->ncolors = an.ncolors;
  s->nnzb_lower = an.nnzb_l;
  s->nnzb_upper = an.nnzb_u;
  s->slices = an.S;
  s->slots_a = an.A.slots();
  s->slots_l = an.L.slots();
  s->slots_u = an.U.slots();
  s->device_bytes = (long long)h->device_bytes;
  s->launches_per_iter = h->per_iter[0];
  s->last_launches = h->last_launches;
  s->factor_ms = h->factor_ms;
  s->analyze_ms = h->analyze_ms;
  s->color_ms = h->color_ms;
  s->color_on_device = h->opt.color_on_device && h->opt.device >= 0 && h->opt.coloring == 0;
  for (int p = 0; p < 2; ++p) {
    s->ring_stages[p] = h->sweep[0][p][0].stage.ring_ns;
    s->ring_stage_bytes[p] = h->sweep[0][p][0].stage.ring_stride;
    s->apply_smem_bytes[p] = h->sweep[0][p][0].stage_bytes;
  }
  for (int p = 0; p < 2; ++p) {
    const double sv = p ? 4.0 : 8.0, sx = sv, si = 4.0;
    const double nb = an.nb, n = 3.0 * an.nb;
    const double nlu = (double)an.nnzb_l + an.nnzb_u;
    s->alg_bytes_spmv[p] = an.nnzb * (9 * sv + si) + (nb + 1) * si + 2 * n * sx;
    s->alg_bytes_ilu[p] = nlu * (9 * sv + si) + 2 * (nb + 1) * si + nb * 9 * sv + 4 * n * sx;
    s->alg_bytes_iter[p] = iter_bytes(h, sv, sx).total();
  }
  return GBILU_OK;
}

int gbilu_dot_check(void *handle, int n, const float *x, const float *y, double *dot_df,
                    double *dot_fp64) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h || n <= 0 || !x || !y) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  if (h->opt.device < 0) return h->fail(GBILU_NO_DEVICE, "host-only handle cannot run the check");
  if (!h->with_32) return h->fail(GBILU_BAD_INPUT, "the FP32 dot check needs GBILU_MIXED");
  if (n > 3 * h->an.nb) return h->fail(GBILU_BAD_INPUT, "n exceeds 3*nb");
  CK(cudaSetDevice(h->opt.device));
  Ctl *c = h->ctl.p + 1;   // the spare control block
  k_ctl_init<<<1, 32, 0, h->st>>>(c, 0.0, 0, 0, 0ull);
  CK(cudaMemcpyAsync(h->v32.r.p, x, n * sizeof(float), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(h->v32.s.p, y, n * sizeof(float), cudaMemcpyHostToDevice, h->st));
  double out[2];
  for (int mode = 0; mode < 2; ++mode) {
    k_dot_check<<<reduce_grid(h, n), kThreads, 0, h->st>>>(c, n, h->v32.r.p, h->v32.s.p, mode,
                                                            h->partials.p);
    CK(cudaMemcpyAsync(h->h_ctl, c, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    out[mode] = h->h_ctl->dots[0];
  }
  CK(last_error(h));
  if (dot_df) *dot_df = out[0];
  if (dot_fp64) *dot_fp64 = out[1];
  return GBILU_OK;
}

int gbilu_wait_probe(void *handle, int mode, int *bar_fail, int *status, double *ms) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h || mode < 0 || mode > 2) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  if (h->opt.device < 0) return h->fail(GBILU_NO_DEVICE, "host-only handle cannot run the probe");
  if (mode == 2) {
    if (!h->small_grid[0] && !h->small_grid[1])
      return h->fail(GBILU_BAD_INPUT, "solves of this handle do not run in one launch");
    h->small_probe = true;
    if (bar_fail) *bar_fail = 0;
    if (status) *status = GBILU_OK;
    if (ms) *ms = 0.0;
    return GBILU_OK;
  }
  CK(cudaSetDevice(h->opt.device));
  Ctl *c = h->ctl.p + 1;   // the spare control block: the solve state stays as it is
  k_ctl_init<<<1, 32, 0, h->st>>>(c, 0.0, 0, 0, 0ull);
  const unsigned long long sent = 0x7ff4a5a5a5a5a5a5ull;   // the data-ordered steps' sentinel
  CK(cudaMemcpyAsync(h->io64.p, &sent, sizeof sent, cudaMemcpyHostToDevice, h->st));
  CK(cudaEventRecord(h->e0, h->st));
  k_wait_probe<<<2, 32, 0, h->st>>>(c, mode, h->io64.p);
  CK(cudaEventRecord(h->e1, h->st));
  CK(cudaMemcpyAsync(h->h_ctl, c, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, h->e0, h->e1));
  if (bar_fail) *bar_fail = h->h_ctl->bar_fail;
  if (status) *status = h->h_ctl->status;
  if (ms) *ms = t;
  return GBILU_OK;
}

int gbilu_device_order(void *handle, int *order) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h || !order) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  for (int d = 0; d < h->an.nb; ++d) order[d] = h->an.perm[h->an.dperm[d]];
  return GBILU_OK;
}

int gbilu_schedule(void *handle, int transpose, int cap, int *nsteps, int *steps) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  if (!h->analyzed) return h->fail(GBILU_NOT_READY, "gbilu_analyze has not been called");
  const std::vector<Phase> st = make_steps(h->an, transpose != 0);
  if (nsteps) *nsteps = (int)st.size();
  for (int q = 0; q < (int)st.size() && q < cap && steps; ++q) {
    const Phase &P = st[q];
    // every step starts at a slice edge and ends with a grid barrier, a CTA
    // barrier when it and the next step run on CTA 0 alone, or none when
    // both are small (staged: the next step waits for the values it reads)
    const int v[13] = {P.row0, P.nrows, P.slice0, 0, P.mat, P.has_d, P.own_y, P.nbr_hat,
                       P.src_rows, P.to_y, P.final0, P.final_d,
                       P.flow_after ? 3 : P.local_after ? 2 : 1};
    memcpy(steps + 13 * q, v, sizeof v);
  }
  return GBILU_OK;
}

int gbilu_ilu_trace(void *handle, int fp32, int transpose, double *us, int *rows, int cap,
                    int *nphases) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (fp32 && !h->with_32) return h->fail(GBILU_BAD_INPUT, "FP32 trace needs GBILU_MIXED");
  if (h->an.ncolors > kMaxPhases / 2) return h->fail(GBILU_BAD_INPUT, "too many colors to trace");
  CK(cudaSetDevice(h->opt.device));
  const int t = transpose ? 1 : 0;
  const PhaseList &pl = h->sweep[0][fp32 ? 1 : 0][t].phases;
  const int n = 3 * h->an.nb;
  CK(cudaMemsetAsync(h->v64.p.p, 0, n * sizeof(double), h->st));
  if (h->with_32) CK(cudaMemsetAsync(h->v32.p.p, 0, n * sizeof(float), h->st));
  for (int rep = 0; rep < 2; ++rep) {   // the second, warm run is reported
    k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, 0.0, 0, 0, 0ull);
    if (fp32) {
      Ops<float, float> o = make_ops<float, float>(h, t != 0);
      CK(cudaMemsetAsync(h->v32.ph.p, 0, n * sizeof(float), h->st));
      CK(launch_coop(h, h->st, o, (const float *)h->v32.p.p, h->v32.ph.p, 1));
    } else {
      Ops<double, double> o = make_ops<double, double>(h, t != 0);
      CK(cudaMemsetAsync(h->v64.ph.p, 0, n * sizeof(double), h->st));
      CK(launch_coop(h, h->st, o, (const double *)h->v64.p.p, h->v64.ph.p, 1));
    }
  }
  CK(cudaMemcpyAsync(h->h_ctl, h->ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(last_error(h));
  if (nphases) *nphases = pl.n;
  for (int q = 0; q < pl.n && q < cap; ++q) {
    if (us) us[q] = (h->h_ctl->phase_ns[q + 1] - h->h_ctl->phase_ns[q]) * 1e-3;
    if (rows) rows[q] = pl.p[q].nrows;
  }
  return GBILU_OK;
}

int gbilu_bench_kernel(void *handle, int which, int reps, double *avg_ms, double *alg_bytes,
                       int *launches_out) {
  Handle *h = static_cast<Handle *>(handle);
  if (!h) return GBILU_BAD_INPUT;
  int rc = check_solve_ready(h);
  if (rc) return rc;
  if (which < 0 || which > 15 || reps <= 0) return h->fail(GBILU_BAD_INPUT, "bad kernel id or reps");
  const bool fp32 = which == 2 || which == 3 || (which >= 9 && which != 14);
  if (fp32 && !h->with_32) return h->fail(GBILU_BAD_INPUT, "FP32 kernels need GBILU_MIXED");
  CK(cudaSetDevice(h->opt.device));
  gbilu_stats st;
  gbilu_get_stats(h, &st);
  const int nb = h->an.nb, n = 3 * nb, g = grid_for(h, n);
  int launches = 0;
  k_ctl_init<<<1, 32, 0, h->st>>>(h->ctl.p, 0.0, 0, 0, 0ull);
  // inputs: a fixed pseudo-random vector in the permuted numbering
  std::vector<double> x(n);
  uint64_t z = 0x9e3779b97f4a7c15ull;
  for (int i = 0; i < n; ++i) {
    z ^= z << 13; z ^= z >> 7; z ^= z << 17;
    x[i] = (double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  }
  CK(cudaMemcpyAsync(h->v64.p.p, x.data(), n * sizeof(double), cudaMemcpyHostToDevice, h->st));
  if (h->with_32) k_scale_convert<<<g, kThreads, 0, h->st>>>(n, 1.0, h->v64.p.p, h->v32.p.p);
  if (which >= 4) {
    // every work vector of the iteration holds its own pseudo-random data,
    // so that the dots and norms are nonzero and no kernel stops the run
    Vecs<double> &w = h->v64;
    std::vector<double> xv(n);
    int k = 0;
    for (DevBuf<double> *b : {&w.x, &w.r, &w.rt, &w.ph, &w.v, &w.s, &w.sh, &w.t, &w.y, &w.base}) {
      ++k;
      for (int i = 0; i < n; ++i) {
        z ^= z << 13; z ^= z >> 7; z ^= z << 17;
        xv[i] = ((double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5) * k;
      }
      CK(cudaMemcpyAsync(b->p, xv.data(), n * sizeof(double), cudaMemcpyHostToDevice, h->st));
      CK(cudaStreamSynchronize(h->st));
    }
    if (h->with_32) {
      Vecs<float> &f = h->v32;
      DevBuf<double> *src[10] = {&w.x, &w.r, &w.rt, &w.ph, &w.v, &w.s, &w.sh, &w.t, &w.y, &w.base};
      DevBuf<float> *dst[10] = {&f.x, &f.r, &f.rt, &f.ph, &f.v, &f.s, &f.sh, &f.t, &f.y, &f.base};
      for (int j = 0; j < 10; ++j)
        k_scale_convert<<<g, kThreads, 0, h->st>>>(n, 1.0, src[j]->p, dst[j]->p);
    }
  }
  // the iteration's kernels as they run: 4-8 FP64, 9-13 FP32 (SpMV with the
  // alpha dot, SpMV with the omega dots, update_s, update_r, update_p) and
  // the apply, 14 FP64, 15 FP32, with solver scalars that never stop the run
  const int kind = which >= 14 ? 3 : which >= 9 ? which - 5 : which;
  if (which >= 4) k_ctl_bench<<<1, 32, 0, h->st>>>(h->ctl.p);
  const int gr = reduce_grid(h, n);
  auto run = [&](int &l) {
    if (which >= 9 && fp32) {
      iter_kernel<float, float>(h, kind, make_ops<float, float>(h, false), n, g, gr, l);
    } else if (which >= 4) {
      iter_kernel<double, double>(h, kind, make_ops<double, double>(h, false), n, g, gr, l);
    } else if (which == 0) {
      Ops<double, double> o = make_ops<double, double>(h, false);
      spmv<double, double, SPMV_PLAIN>(h, h->st, o, h->v64.p.p, h->v64.v.p, nullptr, l);
    } else if (which == 1) {
      Ops<double, double> o = make_ops<double, double>(h, false);
      apply_prec(h, h->st, o, h->v64.p.p, h->v64.ph.p, l);
    } else if (which == 2) {
      Ops<float, float> o = make_ops<float, float>(h, false);
      spmv<float, float, SPMV_PLAIN>(h, h->st, o, h->v32.p.p, h->v32.v.p, nullptr, l);
    } else {
      Ops<float, float> o = make_ops<float, float>(h, false);
      apply_prec(h, h->st, o, h->v32.p.p, h->v32.ph.p, l);
    }
  };
  // the small steps beside update_s and update_p wait for values that
  // update_r has preset: it runs before each, and its own time is taken off
  const bool preset = !fp32 && (kind == 6 || kind == 8) && which >= 4 && reduced_run(h, false) &&
                      flow_run<double>(h, false);
  int warm = 0;
  auto timed = [&](bool with_preset, bool with_run, float &ms) -> int {
    auto pass = [&](int &l) {
      if (with_preset)
        iter_kernel<double, double>(h, 7, make_ops<double, double>(h, false), n, g, gr, warm);
      if (with_run) run(l);
    };
    for (int i = 0; i < 3; ++i) pass(warm);
    CK(cudaStreamSynchronize(h->st));
    CK(cudaEventRecord(h->e0, h->st));
    for (int i = 0; i < reps; ++i) pass(launches);
    CK(cudaEventRecord(h->e1, h->st));
    CK(cudaEventSynchronize(h->e1));
    CK(last_error(h));
    CK(cudaEventElapsedTime(&ms, h->e0, h->e1));
    return GBILU_OK;
  };
  float ms = 0, preset_ms = 0;
  if ((rc = timed(preset, true, ms))) return rc;
  if (preset && (rc = timed(true, false, preset_ms))) return rc;
  if (avg_ms) *avg_ms = (ms - preset_ms) / reps;
  if (alg_bytes) {
    const double sx = fp32 ? 4.0 : 8.0;
    const IterBytes ib = iter_bytes(h, sx, sx);
    const double by[6] = {ib.apply, ib.spmv, ib.spmv, ib.update_s, ib.update_r, ib.update_p};
    *alg_bytes = which >= 4 ? by[kind - 3]
                            : (which == 0 || which == 2) ? st.alg_bytes_spmv[which / 2]
                                                         : st.alg_bytes_ilu[which / 2];
  }
  if (launches_out) *launches_out = launches / reps;
  return GBILU_OK;
}

const char *gbilu_status_string(int s) {
  switch (s) {
    case GBILU_OK: return "ok";
    case GBILU_MAXIT: return "maximum iterations reached";
    case GBILU_ALREADY_CONVERGED: return "initial residual already below the bound";
    case GBILU_BREAKDOWN: return "BiCGSTAB breakdown";
    case GBILU_NONFINITE: return "non-finite residual";
    case GBILU_TIMEOUT: return "device time budget exceeded";
    case GBILU_BAD_INPUT: return "bad input";
    case GBILU_SINGULAR: return "singular diagonal block";
    case GBILU_CUDA_ERROR: return "CUDA error";
    case GBILU_NOT_READY: return "call order";
    case GBILU_NO_DEVICE: return "host-only handle";
    default: return "unknown status";
  }
}

const char *gbilu_last_error(void *handle) {
  Handle *h = static_cast<Handle *>(handle);
  return h ? h->err.c_str() : "null handle";
}

}  // extern "C"
