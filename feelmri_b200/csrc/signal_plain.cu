// Plain CUDA-core forms of Signal (FP32 drop-in and FP64), for samples whose
// wave vectors do not factor (signal_gemm.cu takes the others).
//
// Restates Signal<T> (cpp/feelmri/MRI.cpp:38-159 with motion, :196-298
// without): for every sample s of run g (time t_g)
//   K[s, v] = sum_n exp(i * (-2pi k_s . r_n(t_g) + phi_n t_g)) * MM[n, v] * exp(-t_g / T2_n)
// with MM = M * Mxy and 2pi built from a float-rounded pi (MRI.h:13, MRI.cpp:73).
// The FP64 form sums the phase in radians and takes sin/cos of that, as the
// reference does (MRI.cpp:138-146); the FP32 form sums it in FP64 cycles and
// reduces it exactly (cycles.cuh).  One thread block covers up to 256 samples of
// one run and sweeps a node range staged in shared memory; the per-run node
// quantities (moved position, phase offset, decayed weight) are formed once per
// tile and node.  Node ranges may be split over blocks; partial sums are then added
// in a fixed order.
#include <algorithm>

#include "cycles.cuh"
#include "signal_common.cuh"
#include "signal_gemm.cuh"

namespace fm {

template <typename T>
struct PlainDev {
  int64_t N, S, V;
  const T *kx, *ky, *kz;
  const T *r0, *phi, *T2;
  const T *MM;  // (N, V) complex interleaved
  MotionDev md;
  const float *weights;   // (n_runs, slots) TERMS motion weights
  const T *table;         // TABLE motion (n_runs, N, 3) in T
  const int2 *tiles;      // (run, first sample within it)
  const int *run_start;
  const int *n_tiles;     // device: number of tiles
  const double *run_t;
  int64_t chunk;          // nodes per split
  int splits;
  T *out;                 // (S, V) complex or partials (splits, S, V)
  T two_pi;
};

constexpr int kPlainNodes = 128;            // nodes staged at a time
constexpr int kPlainFold64 = 512;           // nodes in one FP64 sum
constexpr int kPlainBlocks = 4 * kSmCount;  // blocks sharing the tiles: what an SM holds in FP32

// FP64.  Bound by the FP64 pipe's latency in sincos, so by the warps there:
// BLOCKS = 2 of them an SM.  Left to itself the compiler takes more than 128
// registers at two columns and up, and half the blocks: 5,003 nodes x 64 runs x 300
// samples x 2 columns on a B200 1053 us, 787 us with two.  BLOCKS = 1 where all
// blocks have an SM to themselves: they are dealt to the chip's unequal parts in
// equal shares, so that 128 of them would put two on some SMs (8 columns, 100,003
// nodes: 592 us, 877 us with two).  One column fits two blocks either way.
template <int VMAX, int BLOCKS>
__global__ void __launch_bounds__(kPlainThreads, BLOCKS) signal_plain_kernel(PlainDev<double> p, int v0,
                                                                            bool either) {
  __shared__ double4 s_pos[kPlainNodes];         // moved x, y, z and phi * t
  __shared__ double s_w[kPlainNodes][2 * VMAX];  // decayed M * Mxy columns v0 .. v0 + VMAX

  const int n_tiles = *p.n_tiles;
  const int64_t items = (int64_t)n_tiles * p.splits;
  if (either && (items <= kSmCount) != (BLOCKS == 1)) return;  // the other instance's
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const int split = (int)(item / n_tiles), tile = (int)(item - (int64_t)split * n_tiles);
    __syncthreads();  // the previous tile's readers of s_pos / s_w are done
    const int g = p.tiles[tile].x;
    const int s_begin = p.run_start[g] + p.tiles[tile].y, s = s_begin + threadIdx.x;
    const bool in = (int)threadIdx.x < p.run_start[g + 1] - s_begin;  // (s itself may pass 2^31)
    const double tg = p.run_t[g];
    const int nv = (int)min((int64_t)VMAX, p.V - v0);
    // kx_ = two_pi * kloc[0](i,j,k)   (MRI.cpp:138-140)
    const double kx = in ? p.two_pi * p.kx[s] : 0.0;
    const double ky = in ? p.two_pi * p.ky[s] : 0.0;
    const double kz = in ? p.two_pi * p.kz[s] : 0.0;
    double acc_r[VMAX], acc_i[VMAX];
#pragma unroll
    for (int v = 0; v < VMAX; ++v) acc_r[v] = acc_i[v] = 0.0;

    const int64_t n_begin = (int64_t)split * p.chunk;
    const int64_t n_end = min(p.N, n_begin + p.chunk);
    const float *wrun = p.weights ? p.weights + (int64_t)g * p.md.slots : nullptr;
    double *dst = p.out + ((int64_t)split * p.S * p.V + (int64_t)s * p.V + v0) * 2;
    for (int64_t nb = n_begin;; nb += kPlainNodes) {
      // a sum of kPlainFold64 nodes in registers at a time, then added to the output
      if (nb >= n_end || (nb > n_begin && (nb - n_begin) % kPlainFold64 == 0)) {
        const bool first = nb - n_begin <= kPlainFold64;
#pragma unroll
        for (int v = 0; v < VMAX; ++v) {
          if (in && v < nv) {
            dst[2 * v + 0] = first ? acc_r[v] : dst[2 * v + 0] + acc_r[v];
            dst[2 * v + 1] = first ? acc_i[v] : dst[2 * v + 1] + acc_i[v];
          }
          acc_r[v] = acc_i[v] = 0.0;
        }
        if (nb >= n_end) break;
      }
      const int cnt = (int)min((int64_t)kPlainNodes, n_end - nb);
      __syncthreads();
      for (int j = threadIdx.x; j < cnt; j += kPlainThreads) {
        const int64_t n = nb + j;
        double x = p.r0[3 * n + 0], y = p.r0[3 * n + 1], z = p.r0[3 * n + 2];
        if (p.md.kind == FM_MOTION_TERMS) {
          float dx, dy, dz;
          motion_disp(p.md, wrun, n, p.N, dx, dy, dz);
          x = x + (double)dx; y = y + (double)dy; z = z + (double)dz;
        } else if (p.table) {
          const double *d = p.table + ((int64_t)g * p.N + n) * 3;
          x = x + d[0]; y = y + d[1]; z = z + d[2];
        }
        double4 pp;
        pp.x = x; pp.y = y; pp.z = z;
        pp.w = p.phi[n] * tg;                    // phi_off (MRI.cpp:124)
        s_pos[j] = pp;
        const double invT2 = 1.0 / p.T2[n];
        const double decay = exp(-tg * invT2);   // T2_decay (MRI.cpp:127)
        const double *mm = p.MM + (n * p.V + v0) * 2;
#pragma unroll
        for (int v = 0; v < VMAX; ++v) {
          s_w[j][2 * v + 0] = (v < nv) ? mm[2 * v + 0] * decay : 0.0;
          s_w[j][2 * v + 1] = (v < nv) ? mm[2 * v + 1] * decay : 0.0;
        }
      }
      __syncthreads();
      for (int j = 0; j < cnt; ++j) {
        const double4 pp = s_pos[j];
        // phase = -kx_ x - ky_ y - kz_ z + phi_off   (MRI.cpp:143-146)
        const double ph = fma(-kz, pp.z, fma(-ky, pp.y, -kx * pp.x)) + pp.w;
        double sn, cs;
        sincos(ph, &sn, &cs);
#pragma unroll
        for (int v = 0; v < VMAX; ++v) {
          const double wr = s_w[j][2 * v + 0], wi = s_w[j][2 * v + 1];
          acc_r[v] = fma(cs, wr, fma(-sn, wi, acc_r[v]));
          acc_i[v] = fma(cs, wi, fma(sn, wr, acc_i[v]));
        }
      }
    }

  }  // tiles
}

// FP32: two samples per thread, their phases in FP64 cycles.  A phase is three
// multiply-adds on the FP64 pipe,
// which the rest leaves idle, and its reduction exact (cycles.cuh), where the
// reference rounds the phase in radians to FP32; what comes after is FP32 as
// there.  Bound by issue: per sample-node some 40 instructions for the phase and
// its sin/cos and 4 a column, 75% of the issue rate.  20,011 nodes x 128 runs x
// 255 samples x 8 columns, a call on a B200: 3117 us with sincosf of a rounded phase,
// one sample per thread and tiles dealt out split by split, 1900 us now.
constexpr int kPlain32Threads = 128;
constexpr int kPlainFold = 2048;  // nodes in one sum: a longer one is the largest error of the form
template <int VMAX>
__global__ void __launch_bounds__(kPlain32Threads, 4) signal_plain32_kernel(PlainDev<float> p, int v0) {
  __shared__ double4 s_pos[kPlainNodes];         // moved x, y, z and phi t in cycles
  __shared__ float2 s_w[kPlainNodes][VMAX];  // decayed M * Mxy

  const int n_tiles = *p.n_tiles;
  const int64_t items = (int64_t)n_tiles * p.splits;
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const int split = (int)(item / n_tiles), tile = (int)(item - (int64_t)split * n_tiles);
    __syncthreads();  // the previous tile's readers of s_pos / s_w are done
    const int g = p.tiles[tile].x;
    const int s_begin = p.run_start[g] + p.tiles[tile].y, left = p.run_start[g + 1] - s_begin;
    const int s0 = s_begin + threadIdx.x, s1 = s0 + kPlain32Threads;
    const bool in0 = (int)threadIdx.x < left, in1 = (int)threadIdx.x + kPlain32Threads < left;  // (s1 may pass 2^31)
    const float tg = (float)p.run_t[g];
    const int nv = (int)min((int64_t)VMAX, p.V - v0);
    // -k in units of 2 pi with a float-rounded pi
    auto scaled = [&](const float *k, int s, bool in) { return in ? -(double)k[s] * kPiRatio : 0.0; };
    const double kx0 = scaled(p.kx, s0, in0), ky0 = scaled(p.ky, s0, in0), kz0 = scaled(p.kz, s0, in0);
    const double kx1 = scaled(p.kx, s1, in1), ky1 = scaled(p.ky, s1, in1), kz1 = scaled(p.kz, s1, in1);
    float2 acc0[VMAX], acc1[VMAX];
    // nodes are rows of a sparse matrix of 32-bit indices
    const int n_begin = (int)((int64_t)split * p.chunk);
    const int n_end = (int)min(p.N, n_begin + p.chunk);
    const float *wrun = p.weights ? p.weights + (int64_t)g * p.md.slots : nullptr;
    // a sum of kPlainFold nodes in registers at a time, then added to the output
    for (int fold = n_begin;;) {
      const int fold_end = fold + min(kPlainFold, n_end - fold);
#pragma unroll
      for (int v = 0; v < VMAX; ++v) acc0[v] = acc1[v] = make_float2(0.f, 0.f);
      for (int nb = fold; nb < fold_end; nb += kPlainNodes) {
        const int cnt = min(kPlainNodes, fold_end - nb);
        __syncthreads();
        for (int j = threadIdx.x; j < cnt; j += kPlain32Threads) {
          const int64_t n = nb + j;
          float x = p.r0[3 * n + 0], y = p.r0[3 * n + 1], z = p.r0[3 * n + 2];
          if (p.md.kind == FM_MOTION_TERMS) {
            float dx, dy, dz;
            motion_disp(p.md, wrun, n, p.N, dx, dy, dz);
            x = x + dx; y = y + dy; z = z + dz;
          } else if (p.table) {
            const float *d = p.table + ((int64_t)g * p.N + n) * 3;
            x = x + d[0]; y = y + d[1]; z = z + d[2];
          }
          double4 pp;
          pp.x = x; pp.y = y; pp.z = z;
          pp.w = (double)p.phi[n] * tg * kInv2Pi;     // phi_off (MRI.cpp:124)
          s_pos[j] = pp;
          const float invT2 = 1.f / p.T2[n];
          const float decay = expf(-tg * invT2);      // T2_decay (MRI.cpp:127)
          const float *mm = p.MM + (n * p.V + v0) * 2;
#pragma unroll
          for (int v = 0; v < VMAX; ++v) {
            const float wr = v < nv ? mm[2 * v + 0] * decay : 0.f, wi = v < nv ? mm[2 * v + 1] * decay : 0.f;
            s_w[j][v] = make_float2(wr, wi);
          }
        }
        __syncthreads();
#pragma unroll 2
        for (int j = 0; j < cnt; ++j) {
          const double4 pp = s_pos[j];
          // phase = -kx_ x - ky_ y - kz_ z + phi_off   (MRI.cpp:143-146)
          float c0, s0n, c1, s1n;
          cis_cycles(fma(kx0, pp.x, fma(ky0, pp.y, fma(kz0, pp.z, pp.w))), c0, s0n);
          cis_cycles(fma(kx1, pp.x, fma(ky1, pp.y, fma(kz1, pp.z, pp.w))), c1, s1n);
#pragma unroll
          for (int v = 0; v < VMAX; ++v) {
            const float2 w = s_w[j][v];
            acc0[v].x = fmaf(c0, w.x, fmaf(-s0n, w.y, acc0[v].x));
            acc0[v].y = fmaf(c0, w.y, fmaf(s0n, w.x, acc0[v].y));
            acc1[v].x = fmaf(c1, w.x, fmaf(-s1n, w.y, acc1[v].x));
            acc1[v].y = fmaf(c1, w.y, fmaf(s1n, w.x, acc1[v].y));
          }
        }
      }

      float2 *dst = reinterpret_cast<float2 *>(p.out) + (int64_t)split * p.S * p.V + v0;
      auto put = [&](float2 &to, float2 sum) {
        if (fold > n_begin) {
          sum.x += to.x;
          sum.y += to.y;
        }
        to = sum;
      };
#pragma unroll
      for (int v = 0; v < VMAX; ++v) {
        if (v < nv && in0) put(dst[(int64_t)s0 * p.V + v], acc0[v]);
        if (v < nv && in1) put(dst[(int64_t)s1 * p.V + v], acc1[v]);
      }
      fold = fold_end;
      if (fold >= n_end) break;
    }
  }  // tiles
}

// out[e] = sum over the node splits of partial[split][e]: eight threads of a
// block each sum every eighth split in order, then their sums in order.  The
// splits are those of the form that worked.
struct SplitCounts {
  int run_cover, slab_cover;
  int splits[3];  // by form
};
constexpr int kReduceLanes = 8, kReduceElems = 32;
template <typename T>
__global__ void __launch_bounds__(kReduceLanes *kReduceElems)
    split_reduce_kernel(const T *__restrict__ part, SplitCounts c, const int *__restrict__ ctl, int64_t count,
                        T *__restrict__ out) {
  __shared__ T sums[kReduceLanes][kReduceElems];
  const int splits = c.splits[prep_form(c.run_cover, c.slab_cover, ctl)];
  if (splits <= 1) return;
  const int lane = threadIdx.x & (kReduceElems - 1), k0 = threadIdx.x / kReduceElems;
  for (int64_t e0 = (int64_t)blockIdx.x * kReduceElems; e0 < count; e0 += (int64_t)gridDim.x * kReduceElems) {
    const int64_t e = e0 + lane;
    T acc = T(0);
    if (e < count)
      for (int k = k0; k < splits; k += kReduceLanes) acc += part[(int64_t)k * count + e];
    __syncthreads();
    sums[k0][lane] = acc;
    __syncthreads();
    if (k0 == 0 && e < count) {
      T s = sums[0][lane];
#pragma unroll
      for (int i = 1; i < kReduceLanes; ++i) s += sums[i][lane];
      out[e] = s;
    }
  }
}

template <typename T, int VMAX>
static void launch_plain(const PlainDev<T> &p, int64_t tiles, int64_t max_tiles, int v0, cudaStream_t st) {
  const int64_t most = max_tiles * p.splits;
  const unsigned grid = (unsigned)(most < kPlainBlocks ? most : kPlainBlocks);
  if constexpr (sizeof(T) == 4) {
    signal_plain32_kernel<VMAX><<<grid, kPlain32Threads, 0, st>>>(p, v0);
    count_launch();
  } else {
    // slabs that are not runs make more tiles than planned, so the device decides
    const bool either = VMAX > 1 && tiles * p.splits <= kSmCount;
    if constexpr (VMAX > 1) {
      if (either) {
        signal_plain_kernel<VMAX, 1><<<grid, kPlainThreads, 0, st>>>(p, v0, true);
        count_launch();
      }
    }
    signal_plain_kernel<VMAX, 2><<<grid, kPlainThreads, 0, st>>>(p, v0, either);
    count_launch();
  }
}

// Split count for slabs cut to `tiles` tiles, within kPartialBytes (`out_bytes` a
// split).
// FP32, an SM holding four blocks: the most tiles that a block takes, over the
// splits, and 1% a split for its partial sums; at least 1024 nodes a split.  128
// tiles go to 592 blocks in 9 splits, 2 for each block and 0.22 of a tile's time; in
// the fewest splits that give every block one (5), it is 0.4.
// FP64, two blocks: the tiles of the fullest SM, whose blocks share its FP64 pipe
// (the first alone leaves a third of it idle), and 0.2% a split; at least 512 nodes.
// 512 tiles of 2,003 nodes are 4 for some SMs in one split, 7 halves in two: 1107 us
// and 1005 us a call (one column).
template <typename T>
static int choose_splits(int64_t tiles, int64_t N, int64_t out_bytes) {
  constexpr bool f64 = sizeof(T) == 8;
  int best = 1;
  double best_cost = 0.0;
  for (int s = 1; s <= 64 && (s == 1 || (N / s >= (f64 ? 512 : 1024) && s * out_bytes <= kPartialBytes)); ++s) {
    double cost;
    if constexpr (f64) {
      const int64_t on_sm = ceil_div(tiles * s, (int64_t)kSmCount);
      cost = (1.5 * (double)(on_sm / 2 * 2) + 2.0 * (double)(on_sm % 2)) / s * (1.0 + 0.002 * s);
    } else {
      cost = (double)ceil_div(tiles * s, (int64_t)kPlainBlocks) / s * (1.0 + 0.01 * s);
    }
    if (s == 1 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

template <typename T>
struct PlainPlan {
  PrepDev prep;
  PrepDev *dev;
  T *partials;
  GemmPlan gemm[2];
  int splits;
  int tile;
  int64_t tiles;  // of slabs that are runs
};

template <typename T>
static void carve_plain(Carve &c, const fm_signal_args *a, PlainPlan<T> &pl) {
  const int64_t S = a->n_ro * a->n_lines * a->n_kz;
  const int64_t N = a->n_nodes, V = a->n_vencs;
  pl.tile = sizeof(T) == 4 ? 2 * kPlain32Threads : kPlainThreads;
  int *ctl = c.take<int>(kCtlWords);
  pl.dev = c.take<PrepDev>(1);
  carve_prep(c, a, pl.tile, false, 0, sizeof(T), ctl, pl.prep);
  pl.tiles = S > 0 ? a->n_ro * ceil_div(a->n_lines * a->n_kz, (int64_t)pl.tile) : 1;
  pl.splits = choose_splits<T>(pl.tiles, N, S * V * 2 * (int64_t)sizeof(T));
  // (the factored form's estimate leaves too few where products are small: 256 of 4
  // rows, 20,011 nodes, FP64, took 3109 us without this bound, 2758 us with it)
  plan_gemm<T>(a, pl.prep, choose_splits<float>(pl.tiles, N, S * V * 2 * (int64_t)sizeof(T)), pl.gemm);
  const int most = std::max(pl.splits, std::max(pl.gemm[0].splits, pl.gemm[1].splits));
  pl.partials = most > 1 ? c.take<T>((size_t)most * S * V * 2) : nullptr;
}

int validate_signal(const fm_signal_args *a, const char *who);

template <typename T>
int signal_plain(fm_ctx *ctx, const fm_signal_args *a, void *ws, size_t ws_bytes) {
  const char *who = sizeof(T) == 4 ? "fm_signal(F32)" : "fm_signal(F64)";
  cudaStream_t st = ctx->stream;
  const int64_t S = a->n_ro * a->n_lines * a->n_kz;
  const int64_t N = a->n_nodes, V = a->n_vencs;
  Carve cv(ws, ws_bytes);
  PlainPlan<T> pl;
  carve_plain<T>(cv, a, pl);
  FM_TRY(carve_ok(cv, who));
  if (S == 0 || V == 0) return FM_OK;
  T *out = static_cast<T *>(a->out);
  if (N == 0) {
    FM_CUDA(cudaMemsetAsync(out, 0, (size_t)S * V * 2 * sizeof(T), st));
    return FM_OK;
  }
  fill_prep(a, pl.prep);
  FM_TRY(launch_prep<T>(a, &pl.prep, 1, pl.dev, st));
  const MotionDev &md = pl.prep.md;
  const int64_t max_tiles = S + S / pl.tile + 1;

  PlainDev<T> p{};
  p.N = N; p.S = S; p.V = V;
  p.kx = static_cast<const T *>(a->kx);
  p.ky = static_cast<const T *>(a->ky);
  p.kz = static_cast<const T *>(a->kz);
  p.r0 = static_cast<const T *>(a->r0);
  p.phi = static_cast<const T *>(a->phi);
  p.T2 = static_cast<const T *>(a->T2);
  p.MM = static_cast<const T *>(pl.prep.MM);
  p.md = md;
  p.weights = (md.kind == FM_MOTION_TERMS) ? pl.prep.weights : nullptr;
  p.table = (a->motion && a->motion->kind == FM_MOTION_TABLE) ? static_cast<const T *>(a->motion->table) : nullptr;
  p.n_tiles = pl.prep.ctl + kCtlTiles;
  p.tiles = pl.prep.tiles;
  p.run_start = pl.prep.start;
  p.run_t = pl.prep.run_t;
  p.splits = pl.splits;
  p.chunk = ceil_div(N, pl.splits);
  p.out = (pl.splits > 1) ? pl.partials : out;
  // two_pi = 2.0 * PI with PI = (float)M_PI   (MRI.h:13, MRI.cpp:73)
  const float pi_f = 3.14159265358979323846f;
  p.two_pi = (T)2.0 * (T)pi_f;

  ScopedTimer timer(ctx, sizeof(T) == 4 ? "signal_f32" : "signal_f64");
  for (int v0 = 0; v0 < V; v0 += 8) {
    const int64_t nv = V - v0;
    if (nv <= 1) launch_plain<T, 1>(p, pl.tiles, max_tiles, v0, st);
    else if (nv <= 2) launch_plain<T, 2>(p, pl.tiles, max_tiles, v0, st);
    else if (nv <= 4) launch_plain<T, 4>(p, pl.tiles, max_tiles, v0, st);
    else launch_plain<T, 8>(p, pl.tiles, max_tiles, v0, st);
    FM_TRY(check_launch("signal_plain_kernel"));
  }
  FM_TRY(launch_gemm<T>(a, pl.prep, pl.gemm, out, pl.partials, st));
  if (pl.partials) {
    const int64_t count = S * V * 2, blocks = ceil_div(count, kReduceElems);
    const SplitCounts c{pl.prep.run_cover, pl.prep.slab_cover, {pl.gemm[0].splits, pl.gemm[1].splits, pl.splits}};
    const unsigned grid = (unsigned)(blocks < 32 * kSmCount ? blocks : 32 * kSmCount);
    split_reduce_kernel<T><<<grid, kReduceLanes * kReduceElems, 0, st>>>(pl.partials, c, pl.prep.ctl, count, out);
    count_launch();
    FM_TRY(check_launch("split_reduce_kernel"));
  }
  return FM_OK;
}

template <typename T>
int signal_plain_errors(fm_ctx *ctx, const fm_signal_args *a, void *ws, size_t ws_bytes) {
  Carve cv(ws, ws_bytes);
  PlainPlan<T> pl;
  carve_plain<T>(cv, a, pl);
  FM_TRY(carve_ok(cv, "fm_signal"));
  return report_errors(pl.prep.ctl, 1, ctx->stream, sizeof(T) == 4 ? "fm_signal(F32)" : "fm_signal(F64)");
}
template int signal_plain_errors<float>(fm_ctx *, const fm_signal_args *, void *, size_t);
template int signal_plain_errors<double>(fm_ctx *, const fm_signal_args *, void *, size_t);

template int signal_plain<float>(fm_ctx *, const fm_signal_args *, void *, size_t);
template int signal_plain<double>(fm_ctx *, const fm_signal_args *, void *, size_t);

template <typename T>
size_t plain_workspace(const fm_signal_args *a) {
  Carve c(nullptr, 0);
  PlainPlan<T> pl;
  carve_plain<T>(c, a, pl);
  return c.used;
}
template size_t plain_workspace<float>(const fm_signal_args *);
template size_t plain_workspace<double>(const fm_signal_args *);

}  // namespace fm
