// Factored CUDA-core forms of Signal (FP32 and FP64).
//
// Where the samples' wave vectors factor, Signal (cpp/feelmri/MRI.cpp:38-159 /
// :196-298) is a dense complex product over the nodes instead of one sin/cos
// per node-sample:
//   K[r, (q, v)] = sum_n A[r, n] B[n, (q, v)]
// * runs as columns (nothing moves): k(i, j, k) = k_run(i) + k_slab(j, k), rows
//   the samples of a slab, q the runs; A = exp(-i 2pi k_slab . r_n),
//   B = exp(-i 2pi k_run . r_n + i phi_n t_q) exp(-t_q / T2_n) (M Mxy)[n, v];
// * slabs: k(j, k) = k_line(j) + k_kz(k) within every run, rows the lines, q the
//   kz values; B = exp(-i 2pi k_kz . r_n) (M Mxy)[n, v] exp(-t / T2_n + i phi_n t).
// Each component of k belongs wholly to one factor (prep_scan_kernel), so the
// factors' phases are exact products of the inputs: no rounding is added.  The
// FP32 form forms phases in FP64, the FP64 form keeps what their rounding leaves
// out, and both reduce them exactly, where the unfactored FP64 form sums them in
// radians as the reference does; sums over the nodes are in the form's type, cut at
// kGemmFold.  2 pi is built from a float-rounded pi (MRI.h:13).
//
// Block: a tile of rows x (q, v) pairs, 8 x 4 (FP64: 4 x 4) per thread, operands
// of 16 nodes at a time in shared memory.  Forming a pair of elements costs some
// 100 instructions, a product of a thread's block with a node 128 multiply-adds:
// issue bounds the FP32 form (1.46 10^9 warp instructions at 66% of the issue
// rate in the flow case below, two thirds of them multiply-adds), the latency of
// forming operands and the set-up of short node ranges the FP64 one.  Plain
// multiply-adds, not packed ones: those need one operand twice in registers,
// which cost as many moves as they save (2.2 ms against 1.9 ms), and one more
// operand stage in shared memory.
//
// Kernel time on a B200, one sin/cos per node-sample (signal_plain_kernel)
// against this: FP32 50,021 nodes x 48 runs x 48 lines x 16 kz x 4 columns with
// flow 6152 us -> 2020 us (the multiply-adds alone take 820 us), FP64 20,011
// nodes x 64 runs x 64 lines 1403 us -> 68 us (multiply-adds 18 us).
#include <algorithm>

#include "cycles.cuh"
#include "signal_common.cuh"
#include "signal_gemm.cuh"

namespace fm {

constexpr int kGemmNodes = 32;  // nodes whose data are formed at a time
constexpr int kGemmStage = 16;  // nodes per operand stage
// Stages summed in registers before their sum is added to the output.  Rounding
// of one long sum is the largest error of the FP32 form: on 200,740 nodes
// 1.4e-5, and 2.5e-6 with the sums cut, for 4% of the time.
constexpr int kGemmFold = 2048 / kGemmStage;
constexpr int kGemmCols = 4;    // columns per thread
constexpr int kGemmSlots = 16 * kGemmCols;
constexpr int kGemmMaxThreads = 256;

template <typename T>
struct GemmType;
template <>
struct GemmType<float> {
  static constexpr int kRows = 8;  // rows per thread
  static constexpr int kRowBytes = 64;  // their factors at a node
  using V2 = float2;
};
template <>
struct GemmType<double> {
  static constexpr int kRows = 4;
  static constexpr int kRowBytes = 64;
  using V2 = double2;
};

template <typename T>
struct GemmDev {
  int64_t N, S, V;
  const T *kx, *ky, *kz, *r0, *phi, *T2;
  const T *MM;  // (N, V) complex interleaved
  MotionDev md;
  const float *weights;
  const T *table;
  const int *ctl;
  const double *run_t;
  int runs;  // runs as columns
  int run_cover, slab_cover;
  int n_lines, n_kz, n_ro;
  int P, C;         // rows and (q, v) columns of one product
  int TR, TC;       // threads along rows and columns of a tile
  int nr, nc;       // tiles along rows and columns
  int splits;
  int64_t chunk;    // nodes per split
  T *out;           // (S, V) complex, or partials (splits, S, V)
};

__device__ inline float exp_of(float x) { return expf(x); }
__device__ inline double exp_of(double x) { return exp(x); }

// Shared memory of a tile.
template <typename T>
struct GemmSmem {
  uint32_t a, b, stage, node, w, krow, kcol, slot, total;
  __host__ __device__ GemmSmem(int TR, int TC, int nv) {
    const int rows = TR * GemmType<T>::kRows, cols = TC * kGemmCols;
    a = 0;  // [node] x FP32: [row / 8][re, im][row % 8]; FP64: [row] complex
    b = kGemmStage * TR * GemmType<T>::kRowBytes;  // [node][slot] complex
    stage = b + kGemmStage * kGemmSlots * 2 * sizeof(T);
    uint32_t off = 2 * stage;
    node = off;  // [2][x, y, z, 1 / T2, phi] of each node
    off += 2 * 5 * kGemmNodes * 8;
    w = off;  // [2][node][v] weights of the tile's columns
    off += 2 * kGemmNodes * nv * 2 * sizeof(T);
    krow = (off + 15) / 16 * 16;  // [x, y, z, and what rounding left of them][row]
    off = krow + 6 * rows * 8;
    kcol = off;  // [x, y, z, their rest, t][q]
    off += 7 * cols * 8;
    slot = off;  // [col] slot of each column
    off += cols;
    total = off;
  }
};

// Column in slot tc + 16 j of the staged factor.  The low bits are mixed so that the threads that
// form the V columns of neighbouring q store to different banks.
__device__ inline int gemm_col(int j, int tc, int TC) {
  const int c = j * TC + tc;
  return TC & 7 ? c : c ^ ((c >> 3) & 7);
}

__device__ inline void lds4(uint32_t addr, float *a) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]) : "r"(addr));
}
__device__ inline void lds2(uint32_t addr, float &a, float &b) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(addr));
}
__device__ inline void lds2(uint32_t addr, double &a, double &b) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(addr));
}

// Register block of a thread: consecutive rows, and the columns that lie in slots
// tc + 16 j of the staged factor.  All offsets but the node's are constants.
template <typename T>
struct GemmAcc;
template <>
struct GemmAcc<float> {
  float re[8][kGemmCols], im[8][kGemmCols];
  __device__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < kGemmCols; ++j) re[i][j] = im[i][j] = 0.f;
  }
  __device__ void node(uint32_t A, uint32_t B) {
    float a[8], c[8], br, bi;
    lds4(A, a);
    lds4(A + 16, a + 4);
    lds4(A + 32, c);
    lds4(A + 48, c + 4);
#pragma unroll
    for (int j = 0; j < kGemmCols; ++j) {
      lds2(B + 128 * j, br, bi);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        re[i][j] = fmaf(a[i], br, re[i][j]);
        im[i][j] = fmaf(a[i], bi, im[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        re[i][j] = fmaf(-c[i], bi, re[i][j]);
        im[i][j] = fmaf(c[i], br, im[i][j]);
      }
    }
  }
  __device__ float2 get(int i, int j) const { return make_float2(re[i][j], im[i][j]); }
};
template <>
struct GemmAcc<double> {
  double re[4][kGemmCols], im[4][kGemmCols];
  __device__ void clear() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < kGemmCols; ++j) re[i][j] = im[i][j] = 0.0;
  }
  __device__ void node(uint32_t A, uint32_t B) {
    double2 a[4], b;
#pragma unroll
    for (int i = 0; i < 4; ++i) lds2(A + 16 * i, a[i].x, a[i].y);
#pragma unroll
    for (int j = 0; j < kGemmCols; ++j) {
      lds2(B + 256 * j, b.x, b.y);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        re[i][j] = fma(a[i].x, b.x, re[i][j]);
        im[i][j] = fma(a[i].x, b.y, im[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        re[i][j] = fma(-a[i].y, b.y, re[i][j]);
        im[i][j] = fma(a[i].y, b.x, im[i][j]);
      }
    }
  }
  __device__ double2 get(int i, int j) const { return make_double2(re[i][j], im[i][j]); }
};

// Phases of two factor elements, k[i0] at node m0 and k[i1] at node m1: sums in
// FP64 (FP32 form), or with what rounding leaves out (FP64 form).
__device__ inline void phase_pair(const double *k, int stride, int i0, int i1, const double *d, int m0, int m1,
                                  double &c0, double &c1) {
  c0 = fma(k[2 * stride + i0], d[2 * kGemmNodes + m0], fma(k[stride + i0], d[kGemmNodes + m0], k[i0] * d[m0]));
  c1 = fma(k[2 * stride + i1], d[2 * kGemmNodes + m1], fma(k[stride + i1], d[kGemmNodes + m1], k[i1] * d[m1]));
}
__device__ inline void phase_pair(const double *k, int stride, int i0, int i1, const double *d, int m0, int m1,
                                  Cycles &c0, Cycles &c1) {
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    c0.add(k[x * stride + i0], k[(x + 3) * stride + i0], d[x * kGemmNodes + m0]);
    c1.add(k[x * stride + i1], k[(x + 3) * stride + i1], d[x * kGemmNodes + m1]);
  }
}

// Row factor of a stage: a thread's elements are pairs of rows at a node, every
// nt-th of the stage.
template <typename T>
__device__ inline void gemm_rows(unsigned char *A, const double *krow, int rows, const double *d, int cnt, int nt) {
  const int per = rows / 2;
  const int dm = nt / per, dr = nt - dm * per;
  int m = threadIdx.x / per, r = threadIdx.x - m * per;
  while (m < cnt) {
    if constexpr (sizeof(T) == 4) {
      float re0, im0, re1, im1;
      const double2 *k = reinterpret_cast<const double2 *>(krow) + r;
      const double2 kx = k[0], ky = k[per], kz = k[2 * per];
      const double x = d[m], y = d[kGemmNodes + m], z = d[2 * kGemmNodes + m];
      const double c0 = fma(kz.x, z, fma(ky.x, y, kx.x * x));
      const double c1 = fma(kz.y, z, fma(ky.y, y, kx.y * x));
      cis_cycles(c0, re0, im0);
      cis_cycles(c1, re1, im1);
      float2 *a = reinterpret_cast<float2 *>(A) + (m * (per >> 2) + (r >> 2)) * 8 + (r & 3);
      a[0] = make_float2(re0, re1);
      a[4] = make_float2(im0, im1);
    } else {
      Cycles c0, c1;
      phase_pair(krow, rows, 2 * r, 2 * r + 1, d, m, m, c0, c1);
      double re0, im0, re1, im1;
      c0.cis(re0, im0);
      c1.cis(re1, im1);
      double2 *a = reinterpret_cast<double2 *>(A) + m * rows + 2 * r;
      a[0] = make_double2(re0, im0);
      a[1] = make_double2(re1, im1);
    }
    m += dm;
    r += dr;
    if (r >= per) {
      r -= per;
      ++m;
    }
  }
}

// Column factor of a stage: the elements of q at two nodes, then its V columns.
// `off` columns of q0 lie before the tile.
template <typename T>
__device__ inline void gemm_cols(unsigned char *B, const double *kcol, const unsigned char *slots, int cols, int n_cols,
                                 int nq, int V, int nv, int off, bool runs, const double *d,
                                 const typename GemmType<T>::V2 *w, int cnt, int nt) {
  constexpr int kPer = 2;
  const int dm = nt / nq, dq = nt - dm * nq;
  int g = threadIdx.x / nq, q = threadIdx.x - g * nq;
  while (g * kPer < cnt) {
    const int m = g * kPer;
    T er[kPer], ei[kPer];
    if constexpr (sizeof(T) == 4) {
      double c0, c1;
      phase_pair(kcol, cols, q, q, d, m, m + 1, c0, c1);
      if (runs) {
        const double u = kcol[6 * cols + q] * kInv2Pi;
        c0 = fma(u, d[4 * kGemmNodes + m], c0);
        c1 = fma(u, d[4 * kGemmNodes + m + 1], c1);
      }
      cis_cycles(c0, er[0], ei[0]);
      cis_cycles(c1, er[1], ei[1]);
    } else {
      Cycles c0, c1;
      phase_pair(kcol, cols, q, q, d, m, m + 1, c0, c1);
      if (runs) {
        c0.add_turn(d[4 * kGemmNodes + m], kcol[6 * cols + q]);
        c1.add_turn(d[4 * kGemmNodes + m + 1], kcol[6 * cols + q]);
      }
      c0.cis(er[0], ei[0]);
      c1.cis(er[1], ei[1]);
    }
    if (runs) {
      const T t = (T)kcol[6 * cols + q];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const T decay = exp_of(-t * (T)d[3 * kGemmNodes + m + k]);
        er[k] *= decay;
        ei[k] *= decay;
      }
    }
    // columns c0 .. c1 of the tile; column c has weight c mod V
    const int c0 = max(q * V - off, 0), c1 = min((q + 1) * V - off, n_cols);
    int i = q == 0 || off == 0 ? 0 : V - off;
    for (int c = c0; c < c1; ++c) {
      const int at = m * kGemmSlots + slots[c];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const typename GemmType<T>::V2 wv = w[(m + k) * nv + i];
        const T br = wv.x * er[k] - wv.y * ei[k], bi = wv.x * ei[k] + wv.y * er[k];
        typename GemmType<T>::V2 o;
        o.x = br;
        o.y = bi;
        reinterpret_cast<typename GemmType<T>::V2 *>(B)[at + k * kGemmSlots] = o;
      }
      if (++i == V) i = 0;
    }
    g += dm;
    q += dq;
    if (q >= nq) {
      q -= nq;
      ++g;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kGemmMaxThreads, 2) signal_gemm_kernel(GemmDev<T> p) {
  // which factoring holds was found on the device; at most one of the two
  // launches of a call works
  if (prep_form(p.run_cover, p.slab_cover, p.ctl) != (p.runs ? kFormRuns : kFormSlabs)) return;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int RT = GemmType<T>::kRows;
  using V2 = typename GemmType<T>::V2;
  const int TR = p.TR, TC = p.TC, rows = RT * TR, cols = kGemmCols * TC;
  const int tid = threadIdx.x, nt = blockDim.x;
  int u = blockIdx.x;
  const int ct = u % p.nc; u /= p.nc;
  const int rt = u % p.nr; u /= p.nr;
  const int split = u % p.splits;
  const int g = u / p.splits;  // run (slabs)
  const int row0 = rt * rows, col0 = ct * cols;
  const int n_rows = min(rows, p.P - row0), n_cols = min(cols, p.C - col0);
  const int V = (int)p.V;
  const int q0 = col0 / V, nq = (col0 + n_cols - 1) / V - q0 + 1;
  const int nv = min(V, n_cols), off = col0 - q0 * V;
  const GemmSmem<T> L(TR, TC, min(V, cols));
  double *node = reinterpret_cast<double *>(smem + L.node);
  double *krow = reinterpret_cast<double *>(smem + L.krow);
  double *kcol = reinterpret_cast<double *>(smem + L.kcol);
  const int Ls = p.n_lines * p.n_kz;
  // a component of k goes with the columns where it varies along them
  const int cm = p.runs ? prep_run_comps(p.ctl) : prep_kz_comps(p.ctl);
  const T *kc[3] = {p.kx, p.ky, p.kz};
  const int64_t s0 = (int64_t)g * Ls;  // first sample of the slab (runs are slabs here)
  // -k float(pi) / pi, split in two
  auto scaled = [&](double *dst, int stride, double k, bool here) {
    const double hi = here ? -k * kPiRatio : 0.0;
    dst[0] = hi;
    dst[3 * stride] = here ? fma(-k, kPiRatio, -hi) - k * kPiRatioLo : 0.0;
  };
  for (int i = tid; i < rows; i += nt) {
    const int r = row0 + min(i, n_rows - 1);
    const int64_t s = p.runs ? r : s0 + (int64_t)r * p.n_kz;
    for (int d = 0; d < 3; ++d) scaled(krow + d * rows + i, rows, (double)kc[d][s], !((cm >> d) & 1));
  }
  for (int i = tid; i < nq; i += nt) {
    const int64_t s = p.runs ? (int64_t)(q0 + i) * Ls : s0 + q0 + i;
    for (int d = 0; d < 3; ++d) scaled(kcol + d * cols + i, cols, (double)kc[d][s], (cm >> d) & 1);
    kcol[6 * cols + i] = p.runs ? p.run_t[q0 + i] : 0.0;
  }
  const double tg = p.runs ? 0.0 : p.run_t[g];
  const float *wrun = p.weights ? p.weights + (int64_t)g * p.md.slots : nullptr;
  const int64_t n_begin = (int64_t)split * p.chunk, n_end = min(p.N, n_begin + p.chunk);
  // data of node block `blk`, by one warp (the warps take turns): moved position,
  // weights, and (runs) 1 / T2 and phi
  auto form_nodes = [&](int blk, int warp) {
    if ((tid >> 5) != warp) return;
    const int lane = tid & 31;
    double *d = node + (blk & 1) * 5 * kGemmNodes + lane;
    V2 *w = reinterpret_cast<V2 *>(smem + L.w) + ((blk & 1) * kGemmNodes + lane) * nv;
    const int64_t n = n_begin + (int64_t)blk * kGemmNodes + lane;
    double x = 0, y = 0, z = 0, f = 0, h = 0;
    T wr = T(0), wi = T(0);
    if (n < n_end) {
      T tx = p.r0[3 * n], ty = p.r0[3 * n + 1], tz = p.r0[3 * n + 2];
      const T phi = p.phi[n], inv = T(1) / p.T2[n];
      if (p.md.kind == FM_MOTION_TERMS) {
        float dx, dy, dz;
        motion_disp(p.md, wrun, n, p.N, dx, dy, dz);
        tx = tx + (T)dx; ty = ty + (T)dy; tz = tz + (T)dz;
      } else if (p.table) {
        const T *t = p.table + ((int64_t)g * p.N + n) * 3;
        tx = tx + t[0]; ty = ty + t[1]; tz = tz + t[2];
      }
      x = (double)tx; y = (double)ty; z = (double)tz;
      if (p.runs) {
        f = (double)inv;
        h = (double)phi;
      } else {
        double re, im;
        Cycles c;
        c.add_turn((double)phi, tg);
        c.cis(re, im);
        const T decay = exp_of(-(T)tg * inv);
        wr = (T)((double)decay * re);
        wi = (T)((double)decay * im);
      }
      const V2 *mm = reinterpret_cast<const V2 *>(p.MM) + n * V;
      int v = off;
#pragma unroll 4
      for (int i = 0; i < nv; ++i) {
        V2 m = mm[v];
        if (!p.runs) {
          const V2 o = m;
          m.x = o.x * wr - o.y * wi;
          m.y = o.x * wi + o.y * wr;
        }
        w[i] = m;
        if (++v == V) v = 0;
      }
    } else {
      for (int i = 0; i < nv; ++i) w[i] = V2{};
    }
    d[0] = x; d[kGemmNodes] = y; d[2 * kGemmNodes] = z; d[3 * kGemmNodes] = f; d[4 * kGemmNodes] = h;
  };
  GemmAcc<T> acc;
  const int tr = tid / TC, tc = tid - tr * TC;
  const bool works = tr < TR;
  unsigned char *slots = smem + L.slot;
  if (works && tr == 0)
#pragma unroll
    for (int j = 0; j < kGemmCols; ++j) slots[gemm_col(j, tc, TC)] = (unsigned char)(tc + 16 * j);
  const int warps = nt >> 5;
  const uint32_t a_at = (uint32_t)__cvta_generic_to_shared(smem + L.a) + tr * GemmType<T>::kRowBytes;
  const uint32_t b_at = (uint32_t)__cvta_generic_to_shared(smem + L.b) + tc * 2 * sizeof(T);
  const int n_stages = (int)ceil_div(max(n_end - n_begin, (int64_t)0), (int64_t)kGemmStage);
  constexpr int kPerBlock = kGemmNodes / kGemmStage;
  static_assert(kPerBlock > 1, "a node block is formed a barrier before its first stage");
  auto nodes_of = [&](int st) { return (int)min((int64_t)kGemmStage, n_end - n_begin - (int64_t)st * kGemmStage); };
  auto form_stage = [&](int st) {
    const int blk = (st / kPerBlock) & 1, m0 = (st % kPerBlock) * kGemmStage, cnt = nodes_of(st);
    const double *d = node + blk * 5 * kGemmNodes + m0;
    const V2 *w = reinterpret_cast<const V2 *>(smem + L.w) + (blk * kGemmNodes + m0) * nv;
    unsigned char *at = smem + (st & 1) * L.stage;
    gemm_rows<T>(at + L.a, krow, rows, d, cnt, nt);
    gemm_cols<T>(at + L.b, kcol, slots, cols, n_cols, nq, V, nv, off, p.runs, d, w, cnt, nt);
  };
  // two operand stages: one is formed while the other is multiplied, so a stage
  // costs one barrier and the warps of a block need not be in step.  Node data
  // are formed one block ahead.
  form_nodes(0, 0);
  __syncthreads();
  if (n_stages > 0) form_stage(0);
  __syncthreads();
  int turn = 0;
  for (int fold = 0; fold == 0 || fold < n_stages; fold += kGemmFold) {
    acc.clear();
    for (int st = fold; st < min(n_stages, fold + kGemmFold); ++st) {
      if (st % kPerBlock == 0 && st + kPerBlock < n_stages) {
        turn = turn + 1 == warps ? 0 : turn + 1;
        form_nodes(st / kPerBlock + 1, turn);
      }
      if (st + 1 < n_stages) form_stage(st + 1);
      if (works) {
        const int cnt = nodes_of(st);
        uint32_t A = a_at + (st & 1) * L.stage, B = b_at + (st & 1) * L.stage;
#pragma unroll 2
        for (int m = 0; m < cnt; ++m) {
          acc.node(A, B);
          A += TR * GemmType<T>::kRowBytes;
          B += kGemmSlots * 2 * sizeof(T);
        }
      }
      __syncthreads();
    }
    if (!works) continue;
    V2 *dst = reinterpret_cast<V2 *>(p.out) + (int64_t)split * p.S * p.V;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = RT * tr + i;
      if (r >= n_rows) continue;
#pragma unroll
      for (int j = 0; j < kGemmCols; ++j) {
        const int c = gemm_col(j, tc, TC);
        if (c >= n_cols) continue;
        const int q = (col0 + c) / V, v = col0 + c - q * V;
        const int64_t s = p.runs ? (int64_t)q * Ls + row0 + r : s0 + (int64_t)(row0 + r) * p.n_kz + q;
        V2 sum = acc.get(i, j);
        if (fold > 0) {
          const V2 before = dst[s * p.V + v];
          sum.x += before.x;
          sum.y += before.y;
        }
        dst[s * p.V + v] = sum;
      }
    }
  }
}

// Tile shape for a product of P rows and C columns: tiles of about equal size,
// at most 16 x 16 threads.
template <typename T>
static void gemm_shape(int64_t P, int64_t C, int64_t V, GemmPlan &g) {
  constexpr int RT = GemmType<T>::kRows;
  const int64_t nr = ceil_div(P, (int64_t)16 * RT), nc = ceil_div(C, (int64_t)16 * kGemmCols);
  g.P = (int)P;
  g.C = (int)C;
  g.TR = (int)ceil_div(ceil_div(P, nr), (int64_t)RT);
  g.TC = (int)ceil_div(ceil_div(C, nc), (int64_t)kGemmCols);
  g.nr = (int)ceil_div(P, (int64_t)g.TR * RT);
  g.nc = (int)ceil_div(C, (int64_t)g.TC * kGemmCols);
  g.threads = (int)(ceil_div((int64_t)g.TR * g.TC, 32) * 32);
  if (g.threads < 64) g.threads = 64;
  g.smem = GemmSmem<T>(g.TR, g.TC, (int)(V < g.TC * kGemmCols ? V : g.TC * kGemmCols)).total;
}

// Node splits: the least estimated time, in operand stages of a block that has
// its SM to itself.  The blocks of an SM share its arithmetic, so their stages
// add up, at a rate that grows with the warps there (latency: 8 / warps on top);
// a block costs about 3 stages to set up and write, and a round of blocks 30 more
// in latency and uneven ends; partial sums are written and read back at some 20 MB
// a stage.  Splits of at least 64 nodes and within 256 MB of partial sums, and at
// least `least`.
static int gemm_splits(const GemmPlan &g, int64_t N, int64_t out_bytes, int least) {
  const int64_t units = (int64_t)g.products * g.nr * g.nc;
  const int64_t per_sm = std::max(1, std::min(65536 / (128 * g.threads), 228 * 1024 / (g.smem + 1024)));
  int best = least;
  double best_cost = 0.0;
  int64_t most = out_bytes > 0 ? kPartialBytes / out_bytes : 1;
  if (most > 512) most = 512;
  for (int s = least; s == least || (s <= most && N / s >= 64); ++s) {
    const int64_t on_sm = ceil_div(units * s, (int64_t)kSmCount);
    const double warps = (double)std::min(on_sm, per_sm) * (g.threads / 32);
    const double cost = (double)on_sm * ((double)N / s / kGemmStage) * (1.0 + 8.0 / warps) +
                        3.0 * (double)on_sm + 30.0 * (double)ceil_div(on_sm, per_sm) +
                        (s > 1 ? 2.0 * s * (double)out_bytes / 2e7 : 0.0);
    if (s == least || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

template <typename T>
void plan_gemm(const fm_signal_args *a, const PrepDev &pr, int least, GemmPlan (&g)[2]) {
  const int64_t V = a->n_vencs, out_bytes = pr.S * V * 2 * (int64_t)sizeof(T);
  g[0] = g[1] = GemmPlan{};
  if (pr.S == 0 || V == 0 || pr.N == 0) return;
  if (pr.run_cover) {
    gemm_shape<T>(pr.Ls, pr.n_ro * V, V, g[0]);
    g[0].products = 1;
  }
  if (pr.slab_cover) {
    gemm_shape<T>(pr.n_lines, pr.n_kz * V, V, g[1]);
    g[1].products = pr.n_ro;
  }
  for (GemmPlan &k : g)
    if (k.products > 0) k.splits = gemm_splits(k, pr.N, out_bytes, least);
}

template <typename T>
int launch_gemm(const fm_signal_args *a, const PrepDev &pr, const GemmPlan (&g)[2], T *out, T *partials,
                cudaStream_t st) {
  for (int k = 0; k < 2; ++k) {
    if (g[k].products == 0) continue;
    GemmDev<T> p{};
    p.N = pr.N; p.S = pr.S; p.V = pr.V;
    p.kx = static_cast<const T *>(a->kx);
    p.ky = static_cast<const T *>(a->ky);
    p.kz = static_cast<const T *>(a->kz);
    p.r0 = static_cast<const T *>(a->r0);
    p.phi = static_cast<const T *>(a->phi);
    p.T2 = static_cast<const T *>(a->T2);
    p.MM = static_cast<const T *>(pr.MM);
    p.md = pr.md;
    p.weights = pr.md.kind == FM_MOTION_TERMS ? pr.weights : nullptr;
    p.table = (a->motion && a->motion->kind == FM_MOTION_TABLE) ? static_cast<const T *>(a->motion->table) : nullptr;
    p.ctl = pr.ctl;
    p.run_t = pr.run_t;
    p.runs = k == 0;
    p.run_cover = pr.run_cover;
    p.slab_cover = pr.slab_cover;
    p.n_lines = pr.n_lines; p.n_kz = pr.n_kz; p.n_ro = pr.n_ro;
    p.P = g[k].P; p.C = g[k].C;
    p.TR = g[k].TR; p.TC = g[k].TC;
    p.nr = g[k].nr; p.nc = g[k].nc;
    p.splits = g[k].splits;
    p.chunk = ceil_div(pr.N, (int64_t)g[k].splits);
    p.out = g[k].splits > 1 ? partials : out;
    const int64_t blocks = (int64_t)g[k].products * g[k].nr * g[k].nc * g[k].splits;
    FM_REQUIRE(blocks < (1LL << 31), FM_ERR_SHAPE, "fm_signal: %lld tiles", (long long)blocks);
    FM_CUDA(cudaFuncSetAttribute(signal_gemm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)GemmSmem<T>(16, 16, 16 * kGemmCols).total));
    signal_gemm_kernel<T><<<(unsigned)blocks, g[k].threads, g[k].smem, st>>>(p);
    count_launch();
    FM_TRY(check_launch("signal_gemm_kernel"));
  }
  return FM_OK;
}

template void plan_gemm<float>(const fm_signal_args *, const PrepDev &, int, GemmPlan (&)[2]);
template void plan_gemm<double>(const fm_signal_args *, const PrepDev &, int, GemmPlan (&)[2]);
template int launch_gemm<float>(const fm_signal_args *, const PrepDev &, const GemmPlan (&)[2], float *, float *,
                                cudaStream_t);
template int launch_gemm<double>(const fm_signal_args *, const PrepDev &, const GemmPlan (&)[2], double *, double *,
                                 cudaStream_t);

}  // namespace fm
