// Shared Signal preprocessing: distinct-time runs, factoring, tiles and the
// sparse product, for all problems of a call at once.
//
// Five launches whatever the number of problems (grid: stretches of work x
// problems), each phase reading what the one before left in the problem's
// scratch:
//   write   descriptors to device memory, control words and slab flags cleared
//   scan    one pass over the samples and over M's pattern: run starts per
//           stretch, which slabs are one run and factor, whether M is diagonal
//   runs    run starts and times, compacted in order; rows of an M of as many
//           entries as rows that is not diagonal
//   items   M Mxy (of such an M or a diagonal one), motion weights, the largest
//           |phi| and |t|, factored runs and tiles counted
//   fill    factored runs and tiles, compacted in order
// These phases are a few microseconds of work each, so launches bound them:
// one chain per problem (33 launches and copies, the scans two each) took
// 238 us of device time for a 3,083-node Signal of 2,048 samples, 58 us of it
// outside the main kernel, and 1.6 ms of a 16-problem batch.
#include <climits>

#include <cub/cub.cuh>

#include "signal_common.cuh"

namespace fm {

constexpr int kPrepThreads = 256;
// Stretches of the samples: enough blocks to fill the SMs; every block of a
// compaction adds up the counts of the stretches before its own.
constexpr int kPrepChunks = 256;

static size_t cub_scan_bytes(int64_t n) {
  size_t b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b, (int *)nullptr, (int *)nullptr, (int)(n > 0 ? n : 1));
  return b;
}

static void carve_csr(Carve &c, int64_t rows, int64_t nnz, Csr &m) {
  m.rowptr = c.take<int>(rows + 1);
  m.fill = c.take<int>(rows + 1);
  m.col = c.take<int>(nnz + 1);
  m.pos = c.take<int>(nnz + 1);
  m.cub_bytes = cub_scan_bytes(rows + 1);
  m.cub_tmp = c.take<char>(m.cub_bytes);
}

void carve_prep(Carve &c, const fm_signal_args *a, int tile, bool tensor_core, int vgroup, size_t real_bytes, int *ctl,
                PrepDev &p) {
  p = PrepDev{};
  p.S = a->n_ro * a->n_lines * a->n_kz;
  p.N = a->n_nodes;
  p.V = a->n_vencs;
  p.n_ro = (int)(p.S > 0 ? a->n_ro : 0);
  p.n_lines = (int)(p.S > 0 ? a->n_lines : 1);
  p.n_kz = (int)(p.S > 0 ? a->n_kz : 1);
  p.Ls = p.n_lines * p.n_kz;
  p.slabs = tensor_core && p.n_kz > 1;
  p.turns = tensor_core;
  p.stat = p.n_ro > 1 && p.Ls > 1 && (a->motion == nullptr || a->motion->kind == FM_MOTION_NONE);
  const int64_t most_cols = 1 << 30;  // columns of a factored product are counted in int
  p.slab_cover = !tensor_core && p.n_kz > 1 && p.n_lines > 1 && p.n_kz * p.V < most_cols;
  p.run_cover = !tensor_core && p.stat && p.n_ro * p.V < most_cols;
  p.tile = tile;
  p.vgroup = vgroup;
  const int64_t want = ceil_div(p.S, 1024);
  p.n_chunks = (int)(want < 1 ? 1 : (want > kPrepChunks ? kPrepChunks : want));
  p.chunk = (int)(ceil_div(ceil_div(p.S, p.n_chunks), kPrepThreads) * kPrepThreads);
  p.ctl = ctl;
  p.slab_bad = c.take<unsigned char>(p.slabs ? p.n_ro : 1);
  p.chunk_starts = c.take<int>(p.n_chunks);
  p.chunk_fac = c.take<int>(p.n_chunks);
  p.chunk_tiles = c.take<int>(p.n_chunks);
  p.start = c.take<int>(p.S + 1);
  p.run_t = c.take<double>(p.S + 1);
  p.frun = c.take<int>(p.slabs ? p.n_ro : 1);
  p.tiles = c.take<int2>(p.S + p.S / tile + 1);
  p.weights = c.take<float>((size_t)(p.S + 1) * motion_slots(a->motion));
  const int64_t groups = vgroup > 0 ? ceil_div(p.V, (int64_t)vgroup) : 1;
  p.MM = c.take<char>((size_t)(vgroup > 0 ? groups * p.N * vgroup : p.N * p.V) * 2 * real_bytes);
  carve_csr(c, a->m_rows, a->m_nnz, p.csr);
}

void fill_prep(const fm_signal_args *a, PrepDev &p) {
  p.diag = a->m_nnz == a->m_rows ? 1 : 0;
  p.table_calls = (a->motion && a->motion->kind == FM_MOTION_TABLE) ? a->motion->table_calls : -1;
  p.kx = a->kx; p.ky = a->ky; p.kz = a->kz; p.t = a->t; p.phi = a->phi;
  p.indptr = a->m_indptr; p.indices = a->m_indices; p.data = a->m_data;
  p.Mxy = a->Mxy;
  p.md = make_motion_dev(a->motion);
}

// ---- write ---------------------------------------------------------------

// Descriptors travel as kernel parameters (at most 4 KB), so the launch
// sequence holds no pointer to host memory and can be captured.
constexpr int kPrepPerWrite = 4096 / sizeof(PrepDev) > 1 ? (4096 - 64) / sizeof(PrepDev) : 1;
struct PrepChunk {
  PrepDev p[kPrepPerWrite];
};

__global__ void prep_write_kernel(const __grid_constant__ PrepChunk c, PrepDev *__restrict__ dst) {
  const PrepDev &p = c.p[blockIdx.x];
  const uint32_t *src = reinterpret_cast<const uint32_t *>(&p);
  uint32_t *d = reinterpret_cast<uint32_t *>(dst + blockIdx.x);
  for (int i = threadIdx.x; i < (int)(sizeof(PrepDev) / 4); i += blockDim.x) d[i] = src[i];
  if (threadIdx.x < kCtlWords) p.ctl[threadIdx.x] = 0;
  if (p.slabs)
    for (int i = threadIdx.x; i < p.n_ro; i += blockDim.x) p.slab_bad[i] = 0;
}

// ---- scan ----------------------------------------------------------------

// Sum over the block's threads, in every thread.
__device__ inline int block_sum(int v) {
  __shared__ int part[kPrepThreads / 32];
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  int s = 0;
#pragma unroll
  for (int i = 0; i < kPrepThreads / 32; ++i) s += part[i];
  return s;
}

// Exclusive prefix of v over the block's threads; `total` the block's sum.
__device__ inline int block_exclusive(int v, int &total) {
  __shared__ int part[kPrepThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  __syncthreads();
  if (lane == 31) part[warp] = inc;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int i = 0; i < kPrepThreads / 32; ++i) {
    if (i < warp) before += part[i];
    total += part[i];
  }
  return before + inc - v;
}

// Sum of counts[0 .. n).
__device__ inline int block_prefix(const int *counts, int n) {
  int v = 0;
  for (int i = threadIdx.x; i < n; i += kPrepThreads) v += counts[i];
  return block_sum(v);
}

// A run starts where t differs from the previous sample (MRI.cpp:109); the
// first sample always starts one.  NaN never equals anything, so every NaN
// sample starts its own run, as in the reference's `t_old == t` test.
template <typename T>
__device__ inline bool starts_run(const T *t, int64_t s) {
  return s == 0 || !(t[s] == t[s - 1]);
}

template <typename T>
__global__ void __launch_bounds__(kPrepThreads) prep_scan_kernel(const PrepDev *__restrict__ probs) {
  const PrepDev &p = probs[blockIdx.y];
  const T *t = static_cast<const T *>(p.t);
  const T *kc[3] = {static_cast<const T *>(p.kx), static_cast<const T *>(p.ky), static_cast<const T *>(p.kz)};
  int flags = 0;
  const int c = blockIdx.x;
  if (c < p.n_chunks) {
    const int64_t s0 = (int64_t)c * p.chunk, s1 = min(p.S, s0 + p.chunk);
    int starts = 0;
    for (int64_t s = s0 + threadIdx.x; s < s1; s += kPrepThreads) {
      const bool first = starts_run(t, s);
      starts += first ? 1 : 0;
      const int i = (int)((unsigned)s / (unsigned)p.Ls), w = (int)s - i * p.Ls;
      if (first != (w == 0)) {
        // slab i is not exactly one run (nor the slab before it, when a run
        // reaches across its end)
        flags |= kFlagRuns;
        if (p.slabs) {
          p.slab_bad[i] = 1;
          if (w == 0) p.slab_bad[i - 1] = 1;
        }
      }
      if (p.stat) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const T k = kc[d][s];
          if (!(k == kc[d][(int64_t)i * p.Ls])) flags |= kFlagInSlab << d;
          if (!(k == kc[d][w])) flags |= kFlagAcross << d;
        }
      }
      if (p.slab_cover) {
        const int j = w / p.n_kz;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const T k = kc[d][s];
          if (!(k == kc[d][(int64_t)i * p.Ls + (int64_t)j * p.n_kz])) flags |= kFlagAlongKz << d;
          if (!(k == kc[d][(int64_t)i * p.Ls + (w - j * p.n_kz)])) flags |= kFlagOverLines << d;
        }
      }
      if (p.slabs) {
        // k(j, k) == kp_j + kq_k exactly, kq the slab's kz offsets
        const int j = w / p.n_kz, k = w - j * p.n_kz;
        const int64_t b = (int64_t)i * p.Ls;
        bool good = true, same = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double q = (double)kc[d][b + k] - (double)kc[d][b];
          good = good && ((double)kc[d][s] == (double)kc[d][b + (int64_t)j * p.n_kz] + q);
          if (j == 0) same = same && (q == (double)kc[d][k] - (double)kc[d][0]);
        }
        if (!good) {
          p.slab_bad[i] = 1;
          flags |= kFlagSlabs;
        }
        if (!same) flags |= kFlagOffsets;
      }
    }
    starts = block_sum(starts);
    if (threadIdx.x == 0) p.chunk_starts[c] = starts;
  }
  if (p.diag) {
    bool diag = true;
    const int64_t stride = (int64_t)gridDim.x * kPrepThreads;
    for (int64_t k = (int64_t)blockIdx.x * kPrepThreads + threadIdx.x; k < p.N; k += stride) {
      diag = diag && p.indices[k] == (int)k && p.indptr[k] == (int)k;
      p.csr.fill[k] = -1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) diag = diag && p.indptr[p.N] == (int)p.N;
    if (!diag) flags |= kFlagNotDiagonal;
  }
  flags = __reduce_or_sync(0xffffffffu, flags);
  if ((threadIdx.x & 31) == 0 && flags) atomicOr(p.ctl + kCtlFlags, flags);
}

// ---- runs ----------------------------------------------------------------

// M Mxy of an M of as many entries as rows that turned out not to be diagonal
// (a permuted or partly empty one), with no launch of its own: the entries of a row
// are linked here, in any order, and summed in that of their positions below.
//   fill: a row's first entry (-1: none)    pos: the entry after an entry
//   col: an entry's column                  rowptr: room for the order of long rows
__device__ inline bool prep_listed(const PrepDev &p) { return p.diag && (p.ctl[kCtlFlags] & kFlagNotDiagonal); }
__device__ inline void prep_link_rows(const PrepDev &p) {
  const Csr &m = p.csr;
  for (int64_t e = (int64_t)blockIdx.x * kPrepThreads + threadIdx.x; e < p.N; e += (int64_t)gridDim.x * kPrepThreads) {
    const int k = (int)e, i = p.indices[k];
    if (i < 0 || i >= p.N) {
      atomicOr(p.ctl + kCtlError, kErrSparseRow);
      continue;
    }
    // the entry's column: the last that starts at or before it (each entry is
    // linked once, whatever indptr holds, so that the lists end)
    int j = k;
    if (p.indptr[j] > k || p.indptr[j + 1] <= k) {
      int lo = 0, hi = (int)p.N;
      while (hi - lo > 1) {
        const int mid = lo + (hi - lo) / 2;
        if (p.indptr[mid] <= k) lo = mid;
        else hi = mid;
      }
      j = lo;
      if (p.indptr[j] > k || p.indptr[j + 1] <= k) continue;
    }
    m.col[k] = j;
    m.pos[k] = atomicExch(m.fill + i, k);
  }
}

template <typename T>
__global__ void __launch_bounds__(kPrepThreads) prep_runs_kernel(const PrepDev *__restrict__ probs) {
  const PrepDev &p = probs[blockIdx.y];
  const T *t = static_cast<const T *>(p.t);
  const int c = blockIdx.x;
  if (prep_listed(p)) prep_link_rows(p);
  if (c >= p.n_chunks) return;
  if (!(p.ctl[kCtlFlags] & kFlagRuns)) {  // run g is slab g
    for (int64_t g = c * kPrepThreads + threadIdx.x; g < p.n_ro; g += p.n_chunks * kPrepThreads) {
      p.start[g] = (int)(g * p.Ls);
      p.run_t[g] = (double)t[g * p.Ls];
    }
    if (c == 0 && threadIdx.x == 0) {
      p.start[p.n_ro] = (int)p.S;
      p.ctl[kCtlRuns] = p.n_ro;
    }
    return;
  }
  int g0 = block_prefix(p.chunk_starts, c);
  const int64_t s0 = (int64_t)c * p.chunk, s1 = min(p.S, s0 + p.chunk);
  for (int64_t sb = s0; sb < s1; sb += kPrepThreads) {
    const int64_t s = sb + threadIdx.x;
    const bool first = s < s1 && starts_run(t, s);
    int total;
    const int g = g0 + block_exclusive(first ? 1 : 0, total);
    if (first) {
      p.start[g] = (int)s;
      p.run_t[g] = (double)t[s];
    }
    g0 += total;
  }
  if (c == p.n_chunks - 1 && threadIdx.x == 0) {
    p.start[g0] = (int)p.S;
    p.ctl[kCtlRuns] = g0;
  }
}

// ---- items ---------------------------------------------------------------

template <typename T>
struct Cplx;
template <>
struct Cplx<float> {
  using type = float2;
};
template <>
struct Cplx<double> {
  using type = double2;
};

// Element of M Mxy for row i, column v from the row's linked entries.  Up to
// kLinkedRow of them are taken in order by looking for the next one each time; a
// longer row's order is written out and sorted by the thread of its first column,
// which forms the others too.  Split-BF16 call of 200,000 rows and 2 columns on a
// B200: 313 us with a diagonal M, 322 us permuted (2979 us with one block of threads
// for the matrix).
constexpr int kLinkedRow = 8;
template <typename T>
__device__ __noinline__ void prep_linked_row(const PrepDev &p, int64_t i, int64_t v) {
  using C = typename Cplx<T>::type;
  const Csr &m = p.csr;
  const T *w = static_cast<const T *>(p.data);
  const C *x = static_cast<const C *>(p.Mxy);
  C *MM = static_cast<C *>(p.MM);
  auto add = [&](C &acc, int k, int64_t col) {
    const C xe = x[(int64_t)m.col[k] * p.V + col];
    acc.x = fma(w[k], xe.x, acc.x);
    acc.y = fma(w[k], xe.y, acc.y);
  };
  const int head = m.fill[i];
  int n = 0;
  for (int k = head; k >= 0 && (n <= kLinkedRow || v == 0); k = m.pos[k]) ++n;
  if (n <= kLinkedRow) {
    C acc{};
    for (int done = 0, last = -1; done < n; ++done) {
      int next = INT_MAX;
      for (int k = head; k >= 0; k = m.pos[k])
        if (k > last && k < next) next = k;
      add(acc, next, v);
      last = next;
    }
    MM[mm_index(i, v, p.N, p.V, p.vgroup)] = acc;
  } else if (v == 0) {
    int *order = m.rowptr + atomicAdd(p.ctl + kCtlOrder, n);
    int at = n;  // the list is about descending
    for (int k = head; k >= 0; k = m.pos[k]) order[--at] = k;
    int gap = 1;  // Shell's sort
    while (gap < n / 3) gap = 3 * gap + 1;
    for (; gap > 0; gap /= 3)
      for (int k = gap; k < n; ++k) {
        const int e = order[k];
        int q = k - gap;
        for (; q >= 0 && order[q] > e; q -= gap) order[q + gap] = order[q];
        order[q + gap] = e;
      }
    for (int64_t u = 0; u < p.V; ++u) {
      C acc{};
      for (int k = 0; k < n; ++k) add(acc, order[k], u);
      MM[mm_index(i, u, p.N, p.V, p.vgroup)] = acc;
    }
  }
}

// A TABLE motion must hold one entry per run: a shorter one would be read past
// its end, so a problem without them is given no work at all (its error word is
// set, and the call reports it).
__device__ inline bool prep_table_mismatch(const PrepDev &p) {
  return p.table_calls >= 0 && p.table_calls != p.ctl[kCtlRuns];
}

// Nothing of the problem is listed: it goes through a factored CUDA-core form as
// a whole, or has no work.
__device__ inline bool prep_unlisted(const PrepDev &p) {
  return prep_table_mismatch(p) || prep_form(p.run_cover, p.slab_cover, p.ctl) != kFormPlain;
}

// Factored runs (fac) and tiles of the others (tiles) that run g opens.
__device__ inline void prep_run_items(const PrepDev &p, int g, bool &fac, int &tiles) {
  const int s0 = p.start[g], len = p.start[g + 1] - s0;
  fac = p.slabs && len == p.Ls && s0 % p.Ls == 0 && !p.slab_bad[s0 / p.Ls];
  tiles = fac ? 0 : (len + p.tile - 1) / p.tile;
}

template <typename T>
__global__ void __launch_bounds__(kPrepThreads) prep_items_kernel(const PrepDev *__restrict__ probs) {
  using C = typename Cplx<T>::type;
  const PrepDev &p = probs[blockIdx.y];
  const int n_runs = p.ctl[kCtlRuns];
  const int64_t tid = (int64_t)blockIdx.x * kPrepThreads + threadIdx.x, stride = (int64_t)gridDim.x * kPrepThreads;
  int phi_max = 0, t_max = 0;
  if (p.turns) {
    // |x| as float bits, which compare as numbers do and NaN above them
    auto size_bits = [](float x) { return __float_as_int(x) & 0x7fffffff; };
    for (int64_t i = tid; i < max(p.N, (int64_t)n_runs); i += stride) {
      const T phi = i < p.N ? static_cast<const T *>(p.phi)[i] : T(0);
      const double t = i < n_runs ? p.run_t[i] : 0.0;
      phi_max = max(phi_max, size_bits((float)phi));
      if (t == t) t_max = max(t_max, size_bits((float)t));
    }
  }
  if (p.diag && !(p.ctl[kCtlFlags] & kFlagNotDiagonal)) {
    const T *m = static_cast<const T *>(p.data);
    const C *x = static_cast<const C *>(p.Mxy);
    C *MM = static_cast<C *>(p.MM);
    for (int64_t e = tid; e < p.N * p.V; e += stride) {
      const int64_t n = e / p.V;
      const C xe = x[e];
      const T mn = m[n];
      C r;
      r.x = fma(mn, xe.x, T(0));
      r.y = fma(mn, xe.y, T(0));
      MM[mm_index(n, e - n * p.V, p.N, p.V, p.vgroup)] = r;
    }
  }
  if (prep_listed(p))
    for (int64_t e = tid; e < p.N * p.V; e += stride) prep_linked_row<T>(p, e / p.V, e - e / p.V * p.V);
  if (p.md.kind == FM_MOTION_TERMS) {
    const int64_t total = (int64_t)n_runs * p.md.slots;
    for (int64_t idx = tid; idx < total; idx += stride) {
      const int64_t g = idx / p.md.slots;
      p.weights[idx] = motion_weight(p.md, (int)(idx - g * p.md.slots), p.run_t[g]);
    }
  }
  if (p.turns) {
    phi_max = __reduce_max_sync(0xffffffffu, phi_max);
    t_max = __reduce_max_sync(0xffffffffu, t_max);
    if ((threadIdx.x & 31) == 0) {
      if (phi_max) atomicMax(p.ctl + kCtlPhi, phi_max);
      if (t_max) atomicMax(p.ctl + kCtlTime, t_max);
    }
  }
  if (tid == 0 && prep_table_mismatch(p)) atomicOr(p.ctl + kCtlError, kErrTableCalls);
  const int c = blockIdx.x;
  if (c >= p.n_chunks) return;
  const int per = (n_runs + p.n_chunks - 1) / p.n_chunks;
  const int64_t g1 = prep_unlisted(p) ? 0 : min((int64_t)n_runs, (int64_t)(c + 1) * per);
  int nf = 0, nt = 0;
  for (int64_t g = (int64_t)c * per + threadIdx.x; g < g1; g += kPrepThreads) {
    bool fac;
    int tiles;
    prep_run_items(p, (int)g, fac, tiles);
    nf += fac ? 1 : 0;
    nt += tiles;
  }
  nf = block_sum(nf);
  nt = block_sum(nt);
  if (threadIdx.x == 0) {
    p.chunk_fac[c] = nf;
    p.chunk_tiles[c] = nt;
  }
}

// ---- fill ----------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(kPrepThreads) prep_fill_kernel(const PrepDev *__restrict__ probs) {
  const PrepDev &p = probs[blockIdx.y];
  const int c = blockIdx.x;
  if (c >= p.n_chunks) return;
  int f0 = block_prefix(p.chunk_fac, c);
  int t0 = block_prefix(p.chunk_tiles, c);
  const int n_runs = p.ctl[kCtlRuns];
  const int per = (n_runs + p.n_chunks - 1) / p.n_chunks;
  const int64_t g1 = prep_unlisted(p) ? 0 : min((int64_t)n_runs, (int64_t)(c + 1) * per);
  for (int64_t gb = (int64_t)c * per; gb < g1; gb += kPrepThreads) {
    const int64_t g = gb + threadIdx.x;
    bool fac = false;
    int tiles = 0, nf, nt;
    if (g < g1) prep_run_items(p, (int)g, fac, tiles);
    const int f = f0 + block_exclusive(fac ? 1 : 0, nf);
    const int k = t0 + block_exclusive(tiles, nt);
    if (fac) p.frun[f] = (int)g;
    for (int i = 0; i < tiles; ++i) p.tiles[k + i] = make_int2((int)g, i * p.tile);
    f0 += nf;
    t0 += nt;
  }
  if (c == p.n_chunks - 1 && threadIdx.x == 0) {
    p.ctl[kCtlFac] = f0;
    p.ctl[kCtlTiles] = t0;
  }
}

int report_errors(const int *ctl, int n, cudaStream_t st, const char *who) {
  std::vector<int> words((size_t)n * kCtlWords);
  FM_CUDA(cudaMemcpyAsync(words.data(), ctl, words.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  FM_CUDA(cudaStreamSynchronize(st));
  for (int i = 0; i < n; ++i) {
    const int h = words[(size_t)i * kCtlWords + kCtlError];
    FM_REQUIRE(!(h & kErrSparseRow), FM_ERR_SHAPE, "%s: sparse M has a row index outside [0, rows)", who);
    FM_REQUIRE(!(h & kErrTableCalls), FM_ERR_SHAPE,
               "%s: TABLE motion must hold one entry per distinct-time run of t", who);
    FM_REQUIRE(!(h & kErrTimeout), FM_ERR_TIMEOUT, "%s: a tensor-core pipeline wait timed out", who);
    FM_REQUIRE(!(h & kErrPhaseRange), FM_ERR_ARG,
               "%s: the split-BF16 form reduces phases k . r in fixed point and needs (|kx|+|ky|+|kz|) * "
               "(|x|+|y|+|z|) below 2^27 cycles for every sample and moved node (or finite positions), and "
               "off-resonance phases phi t below 2^27 cycles; use precision f32 or f64",
               who);
  }
  return FM_OK;
}

// ---- CSC -> CSR in Eigen's accumulation order ---------------------------

__global__ void csr_count_kernel(const int *__restrict__ indices, int64_t nnz, int64_t rows, int *__restrict__ cnt,
                                 int *__restrict__ bad) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  const int i = indices[k];
  if (i < 0 || i >= rows) {
    atomicOr(bad, kErrSparseRow);
    return;
  }
  atomicAdd(cnt + i, 1);
}

__global__ void csr_scatter_kernel(const int *__restrict__ indptr, const int *__restrict__ indices, int64_t cols,
                                   int64_t rows, const int *__restrict__ rowptr, int *__restrict__ fill,
                                   int *__restrict__ col, int *__restrict__ pos) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cols) return;
  for (int k = indptr[j]; k < indptr[j + 1]; ++k) {
    const int i = indices[k];
    if (i < 0 || i >= rows) continue;
    const int slot = atomicAdd(fill + i, 1);
    col[rowptr[i] + slot] = (int)j;
    pos[rowptr[i] + slot] = k;
  }
}

// Entries of a row sorted by CSC position, which orders them by column and,
// inside a column, by storage order: the order Eigen visits them.
__global__ void csr_sort_kernel(const int *__restrict__ rowptr, int64_t rows, int *__restrict__ col,
                                int *__restrict__ pos) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows) return;
  const int b = rowptr[i], e = rowptr[i + 1];
  for (int k = b + 1; k < e; ++k) {
    const int pk = pos[k], ck = col[k];
    int m = k - 1;
    while (m >= b && pos[m] > pk) {
      pos[m + 1] = pos[m];
      col[m + 1] = col[m];
      --m;
    }
    pos[m + 1] = pk;
    col[m + 1] = ck;
  }
}

template <typename T>
__global__ void spmm_kernel(const int *__restrict__ rowptr, const int *__restrict__ col, const int *__restrict__ pos,
                            const T *__restrict__ data, int64_t rows, int64_t V, int vgroup,
                            const typename Cplx<T>::type *__restrict__ Mxy, typename Cplx<T>::type *__restrict__ MM) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * V) return;
  const int64_t i = idx / V, v = idx - (idx / V) * V;
  typename Cplx<T>::type acc;
  acc.x = T(0); acc.y = T(0);
  for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
    const T m = data[pos[k]];
    const typename Cplx<T>::type x = Mxy[(int64_t)col[k] * V + v];
    acc.x = fma(m, x.x, acc.x);
    acc.y = fma(m, x.y, acc.y);
  }
  MM[mm_index(i, v, rows, V, vgroup)] = acc;
}

// MM[i, v] = sum_j M[i, j] * Mxy[j, v] accumulated over j ascending (Eigen's
// column-major sparse x dense product, cpp/feelmri/MRI.cpp:92).
template <typename T>
static int sparse_times_dense(const fm_signal_args *a, const PrepDev &p, cudaStream_t st) {
  const int64_t rows = a->m_rows, cols = a->m_cols, nnz = a->m_nnz, V = a->n_vencs;
  const Csr &m = p.csr;
  FM_CUDA(cudaMemsetAsync(m.fill, 0, (rows + 1) * sizeof(int), st));
  if (nnz > 0) {
    csr_count_kernel<<<(unsigned)ceil_div(nnz, 256), 256, 0, st>>>(a->m_indices, nnz, rows, m.fill,
                                                                   p.ctl + kCtlError);
    count_launch();
    FM_TRY(check_launch("csr_count_kernel"));
  }
  size_t cb = m.cub_bytes;
  FM_CUDA(cub::DeviceScan::ExclusiveSum(m.cub_tmp, cb, m.fill, m.rowptr, (int)(rows + 1), st));
  count_launch();
  FM_CUDA(cudaMemsetAsync(m.fill, 0, (rows + 1) * sizeof(int), st));
  if (cols > 0 && nnz > 0) {
    csr_scatter_kernel<<<(unsigned)ceil_div(cols, 256), 256, 0, st>>>(a->m_indptr, a->m_indices, cols, rows,
                                                                      m.rowptr, m.fill, m.col, m.pos);
    count_launch();
    FM_TRY(check_launch("csr_scatter_kernel"));
    csr_sort_kernel<<<(unsigned)ceil_div(rows, 256), 256, 0, st>>>(m.rowptr, rows, m.col, m.pos);
    count_launch();
    FM_TRY(check_launch("csr_sort_kernel"));
  }
  if (rows * V > 0) {
    using C = typename Cplx<T>::type;
    spmm_kernel<T><<<(unsigned)ceil_div(rows * V, 256), 256, 0, st>>>(
        m.rowptr, m.col, m.pos, static_cast<const T *>(a->m_data), rows, V, p.vgroup, static_cast<const C *>(a->Mxy),
        static_cast<C *>(p.MM));
    count_launch();
    FM_TRY(check_launch("spmm_kernel"));
  }
  return FM_OK;
}

template <typename T>
int launch_prep(const fm_signal_args *probs, const PrepDev *host, int n, PrepDev *dev, cudaStream_t st) {
  if (n == 0) return FM_OK;
  int chunks = 1, wide = 1;
  for (int i = 0; i < n; ++i) {
    if (host[i].n_chunks > chunks) chunks = host[i].n_chunks;
    int64_t w = ceil_div(host[i].N * host[i].V, 2 * kPrepThreads);
    if (w > kPrepChunks) w = kPrepChunks;
    if (w > wide) wide = (int)w;
  }
  if (chunks > wide) wide = chunks;
  for (int i0 = 0; i0 < n; i0 += kPrepPerWrite) {
    PrepChunk c;
    const int k = (n - i0) < kPrepPerWrite ? (n - i0) : kPrepPerWrite;
    for (int i = 0; i < k; ++i) c.p[i] = host[i0 + i];
    prep_write_kernel<<<(unsigned)k, kPrepThreads, 0, st>>>(c, dev + i0);
    count_launch();
    FM_TRY(check_launch("prep_write_kernel"));
  }
  // grids of at most 65535 problems
  for (int i0 = 0; i0 < n; i0 += 65535) {
    const unsigned y = (unsigned)((n - i0) < 65535 ? (n - i0) : 65535);
    const PrepDev *d = dev + i0;
    prep_scan_kernel<T><<<dim3(wide, y), kPrepThreads, 0, st>>>(d);
    count_launch();
    FM_TRY(check_launch("prep_scan_kernel"));
    prep_runs_kernel<T><<<dim3(wide, y), kPrepThreads, 0, st>>>(d);
    count_launch();
    FM_TRY(check_launch("prep_runs_kernel"));
    prep_items_kernel<T><<<dim3(wide, y), kPrepThreads, 0, st>>>(d);
    count_launch();
    FM_TRY(check_launch("prep_items_kernel"));
    prep_fill_kernel<T><<<dim3(chunks, y), kPrepThreads, 0, st>>>(d);
    count_launch();
    FM_TRY(check_launch("prep_fill_kernel"));
  }
  for (int i = 0; i < n; ++i)
    if (!host[i].diag) FM_TRY(sparse_times_dense<T>(&probs[i], host[i], st));
  return FM_OK;
}

template int launch_prep<float>(const fm_signal_args *, const PrepDev *, int, PrepDev *, cudaStream_t);
template int launch_prep<double>(const fm_signal_args *, const PrepDev *, int, PrepDev *, cudaStream_t);

}  // namespace fm
