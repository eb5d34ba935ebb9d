// Finite-element mass assembly and lumping.
//
// Restates MassAssemble<T> (cpp/feelmri/Assemble.cpp:79-116): per element
// the local matrix Me = sum_q (S S^T) |det J| w_q (LocalMassAssemble,
// Assemble.cpp:59-75; J from the tabulated reference gradients, IsoMapping
// Assemble.cpp:16-55), emitted as triplets (elem(i), elem(j), Me(i,j)) in
// element order and combined as Eigen's setFromTriplets does: duplicates
// summed in insertion order, CSC with row indices sorted inside each column.
//
// On the device the triplets of a column are those of the elements around its
// node, a few hundred at most in a mesh.  So the elements are listed by node
// (a counting sort) and one warp per column orders its own triplets by row in
// shared memory, each against all others, ties in insertion order; duplicates
// are neighbours then and are summed in that order.  A column of more triplets
// than a warp holds sends the whole matrix through a stable radix sort on
// (column, row) instead, which takes any mesh.
// Bound by the comparisons (some 90^2 a column of a tetrahedral mesh).
//
// Lumping restates FEMPhantom.mass_matrix(lumped=True)
// (python/feelmri/Phantom.py:395-398): row sums as scipy forms them for a
// CSC matrix (csc @ ones: columns visited in ascending order).  The
// assembled matrix is symmetric entry for entry (S_i S_j == S_j S_i, and
// both entries collect the same elements in the same order), so row i summed
// over ascending columns equals column i summed over ascending rows.
#include <climits>

#include <cub/cub.cuh>

#include "common.cuh"

namespace fm {

constexpr int kMaxNb = 10;

// Triplets that a warp orders: four to ten times what the nodes of a mesh of
// good elements have (24 tetrahedra or 8 hexahedra around a node).
template <int NB>
constexpr int kWarpTriplets = NB <= 5 ? 256 : 512;
constexpr int kColWarps = 4;

// Element matrices, Me(i, j) at vals[(e nb + j) nb + i] so that the entries of a
// column lie together, and each element's place among those of its nodes; `over`
// is set where a node has more elements than a warp orders.
template <typename T, int NB>
__global__ void __launch_bounds__(128) mass_local_kernel(int64_t E, const int *__restrict__ elems, int64_t N,
                                                         const T *__restrict__ nodes, int Q, const T *__restrict__ qw,
                                                         const T *__restrict__ tab, T *__restrict__ vals,
                                                         int *__restrict__ degree, int *__restrict__ place,
                                                         int *__restrict__ bad, int *__restrict__ over) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  T X[NB][3];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    int v = elems[e * NB + i];
    if (v < 0 || v >= N) {
      atomicExch(bad, 1);
      v = 0;
    }
    const int at = atomicAdd(degree + v, 1);
    if (at == kWarpTriplets<NB> / NB) *over = 1;
    place[e * NB + i] = at;
    X[i][0] = nodes[3 * (int64_t)v + 0];
    X[i][1] = nodes[3 * (int64_t)v + 1];
    X[i][2] = nodes[3 * (int64_t)v + 2];
  }
  T Me[NB * NB];
#pragma unroll
  for (int k = 0; k < NB * NB; ++k) Me[k] = T(0);
  for (int q = 0; q < Q; ++q) {
    const T *Sq = tab + (size_t)q * 4 * NB;
    // J(a, c) = sum_i dS_a[i] * X[i][c]   (Assemble.cpp:36-44)
    T J[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const T *dS = Sq + (size_t)(a + 1) * NB;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T s = T(0);
#pragma unroll
        for (int i = 0; i < NB; ++i) s = s + dS[i] * X[i][c];
        J[a][c] = s;
      }
    }
    // Cofactor expansion along the first row (Eigen's 3x3 determinant).
    const T det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                  J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                  J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
    const T adet = det < T(0) ? -det : det;
    const T w = qw[q];
    // Me += (S S^T) * |detJ| * w_q   (Assemble.cpp:72)
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) Me[i * NB + j] = Me[i * NB + j] + ((Sq[i] * Sq[j]) * adet) * w;
  }
  T *out = vals + e * NB * NB;
#pragma unroll
  for (int j = 0; j < NB; ++j)
#pragma unroll
    for (int i = 0; i < NB; ++i) out[j * NB + i] = Me[i * NB + j];
}

// around[start[v] ..]: e nb + j for every element e with node v in place j.
template <int NB>
__global__ void mass_around_kernel(int64_t count, const int *__restrict__ elems, int64_t N,
                                   const int *__restrict__ start, const int *__restrict__ place,
                                   int *__restrict__ around, const int *__restrict__ over) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count || *over) return;
  int v = elems[k];
  if (v < 0 || v >= N) v = 0;
  around[start[v] + place[k]] = (int)k;
}

// One warp per column: its distinct rows, ascending, and the sums of their
// triplets at rows/data[start[c] nb ..], their number in count[c]; or, with
// `lump`, the sum of those.
template <typename T, int NB>
__global__ void __launch_bounds__(32 * kColWarps) mass_columns_kernel(int64_t N, const int *__restrict__ elems,
                                                                      const T *__restrict__ vals,
                                                                      const int *__restrict__ start,
                                                                      const int *__restrict__ around,
                                                                      int *__restrict__ rows_out,
                                                                      T *__restrict__ data_out,
                                                                      int *__restrict__ count, T *__restrict__ lump,
                                                                      const int *__restrict__ over) {
  constexpr int CAP = kWarpTriplets<NB>;
  __shared__ __align__(16) int s_row[kColWarps][CAP], s_sorted[kColWarps][CAP];
  __shared__ __align__(16) T s_val[kColWarps][CAP], s_vsorted[kColWarps][CAP];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t c = (int64_t)blockIdx.x * kColWarps + warp;
  if (c >= N || *over) return;  // (the matrix is sorted then)
  const int first = start[c], d = start[c + 1] - first, m = d * NB;
  int *row = s_row[warp], *sorted = s_sorted[warp];
  T *val = s_val[warp], *vsorted = s_vsorted[warp];
  // the elements around the node in element order
  int *raw = reinterpret_cast<int *>(val), *list = sorted;
  for (int p = lane; p < d; p += 32) raw[p] = around[first + p];
  __syncwarp();
  for (int p = lane; p < d; p += 32) {
    const int k = raw[p];
    int r = 0;
    for (int q = 0; q < d; ++q) r += raw[q] < k ? 1 : 0;
    list[r] = k;
  }
  __syncwarp();
  // triplets in insertion order: by element, row place, column place (an element
  // may hold a node twice)
  for (int t = lane; t < m; t += 32) {
    const int p = t / NB, i = t - p * NB, k = list[p], e = k / NB;
    int p0 = p, p1 = p + 1;
    while (p0 > 0 && list[p0 - 1] / NB == e) --p0;
    while (p1 < d && list[p1] / NB == e) ++p1;
    const int at = p0 * NB + i * (p1 - p0) + (p - p0);
    row[at] = elems[(int64_t)e * NB + i];
    val[at] = vals[(int64_t)k * NB + i];
  }
  for (int t = m + lane; t < ((m + 3) & ~3); t += 32) row[t] = INT_MAX;
  __syncwarp();
  // place of each among all: rows ascending, equal ones as inserted, so an equal
  // row counts where it comes before
  for (int tb = 0; tb < m; tb += 32) {
    const int t = tb + lane, r = t < m ? row[t] : 0;
    const int4 *o = reinterpret_cast<const int4 *>(row);
    int at = 0, q = 0;
    for (; q < tb / 4; ++q)
      at += (o[q].x <= r) + (o[q].y <= r) + (o[q].z <= r) + (o[q].w <= r);
    for (; q < min(tb / 4 + 8, (m + 3) / 4); ++q) {
      const int k = t - 4 * q;  // r + 1 for those before t
      at += (o[q].x < r + (k > 0)) + (o[q].y < r + (k > 1)) + (o[q].z < r + (k > 2)) + (o[q].w < r + (k > 3));
    }
    for (; q < (m + 3) / 4; ++q)
      at += (o[q].x < r) + (o[q].y < r) + (o[q].z < r) + (o[q].w < r);
    if (t < m) {
      sorted[at] = r;
      vsorted[at] = val[t];
    }
  }
  __syncwarp();
  int n = 0;
  for (int tb = 0; tb < m; tb += 32) {
    const int t = tb + lane;
    const bool head = t < m && (t == 0 || sorted[t] != sorted[t - 1]);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    if (head) {
      const int r = sorted[t], u = n + __popc(heads & ((1u << lane) - 1));
      T acc = vsorted[t];
      for (int q = t + 1; q < m && sorted[q] == r; ++q) acc = acc + vsorted[q];
      if (lump) {
        val[u] = acc;
      } else {
        rows_out[(int64_t)first * NB + u] = r;
        data_out[(int64_t)first * NB + u] = acc;
      }
    }
    n += __popc(heads);
  }
  if (lump) {
    __syncwarp();
    if (lane == 0) {
      T acc = T(0);
      for (int u = 0; u < n; ++u) acc = acc + val[u];
      lump[c] = acc;
    }
  } else if (lane == 0) {
    count[c] = n;
  }
}

// Columns from where mass_columns_kernel left them to the matrix.
template <typename T>
__global__ void mass_pack_kernel(int64_t N, int nb, const int *__restrict__ start, const int *__restrict__ indptr,
                                 const int *__restrict__ rows, const T *__restrict__ from, int *__restrict__ indices,
                                 T *__restrict__ data) {
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  if (c >= N) return;
  const int64_t at = (int64_t)start[c] * nb;
  const int o = indptr[c], n = indptr[c + 1] - o;
  for (int u = threadIdx.x & 15; u < n; u += 16) {
    indices[o + u] = rows[at + u];
    data[o + u] = from[at + u];
  }
}

// Triplets in insertion order: (column, row) and where the value lies.
__global__ void mass_triplets_kernel(int64_t K, int nb, const int *__restrict__ elems,
                                     unsigned long long *__restrict__ keys, int *__restrict__ order) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  const int64_t e = k / (nb * nb);
  const int ij = (int)(k - e * nb * nb), i = ij / nb, j = ij - i * nb;
  keys[k] = ((unsigned long long)(unsigned)elems[e * nb + j] << 32) | (unsigned)elems[e * nb + i];
  order[k] = (int)((e * nb + j) * nb + i);
}

__global__ void mass_heads_kernel(const unsigned long long *__restrict__ keys, int64_t K, int *__restrict__ head) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  head[k] = (k == 0 || keys[k] != keys[k - 1]) ? 1 : 0;
}

// One thread per distinct (col, row): its column is counted, and (when
// writing) its duplicates are summed in insertion order (the sort is stable).
template <typename T>
__global__ void mass_collapse_kernel(const unsigned long long *__restrict__ keys, const int *__restrict__ order,
                                     const T *__restrict__ vals, const int *__restrict__ head,
                                     const int *__restrict__ uid, int64_t K, int *__restrict__ indices,
                                     T *__restrict__ data, int *__restrict__ colcount, int write) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K || !head[k]) return;
  const unsigned long long key = keys[k];
  if (colcount) atomicAdd(colcount + (int)(key >> 32), 1);
  if (!write) return;
  T acc = vals[order[k]];
  for (int64_t m = k + 1; m < K && !head[m]; ++m) acc = acc + vals[order[m]];
  const int u = uid[k] - 1;
  if (indices) indices[u] = (int)(key & 0xffffffffULL);
  data[u] = acc;
}

// lumped[c] = sum over the entries of column c in ascending row order.
template <typename T>
__global__ void mass_lump_kernel(const int *__restrict__ indptr, const T *__restrict__ data, int64_t N,
                                 T *__restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  T acc = T(0);
  for (int k = indptr[c]; k < indptr[c + 1]; ++k) acc = acc + data[k];
  out[c] = acc;
}

// Status words of a build.
enum { kMassNnz, kMassBad, kMassOver, kMassWords = 4 };

struct MassPlan {
  void *vals;
  int *degree, *start, *place, *around;  // elements by node
  int *rows;                             // columns before packing, with `data`
  void *data;
  int *colcount, *indptr, *status;
  // radix sort (in the place of around, rows, data)
  unsigned long long *keys_in, *keys_out;
  int *ord_in, *ord_out, *head, *uid;
  void *lump_data;
  void *cub_tmp;
  size_t cub_bytes;
};

static int64_t n_triplets(const fm_mass_args *a) { return a->n_elems * a->nodes_per_elem * a->nodes_per_elem; }

static void carve_mass(Carve &c, const fm_mass_args *a, int is_double, MassPlan &p) {
  const int64_t K = n_triplets(a);
  const size_t tsz = is_double ? sizeof(double) : sizeof(float);
  p.vals = c.take<char>((K + 1) * tsz);
  p.degree = c.take<int>(a->n_nodes + 2);
  p.start = c.take<int>(a->n_nodes + 2);
  p.colcount = c.take<int>(a->n_nodes + 2);
  p.indptr = c.take<int>(a->n_nodes + 2);
  p.status = c.take<int>(kMassWords);
  p.keys_in = c.take<unsigned long long>(K + 1);
  p.keys_out = c.take<unsigned long long>(K + 1);
  p.ord_in = c.take<int>(K + 1);
  p.ord_out = c.take<int>(K + 1);
  p.head = c.take<int>(K + 1);
  p.uid = c.take<int>(K + 1);
  p.lump_data = c.take<char>((K + 1) * tsz);
  p.place = p.head;
  p.around = p.uid;
  p.rows = p.ord_out;
  p.data = p.keys_out;
  size_t b1 = 0, b2 = 0, b3 = 0;
  const int Ki = (int)(K > 0 ? K : 1);
  cub::DeviceRadixSort::SortPairs(nullptr, b1, (unsigned long long *)nullptr, (unsigned long long *)nullptr,
                                  (int *)nullptr, (int *)nullptr, Ki);
  cub::DeviceScan::InclusiveSum(nullptr, b2, (int *)nullptr, (int *)nullptr, Ki);
  cub::DeviceScan::ExclusiveSum(nullptr, b3, (int *)nullptr, (int *)nullptr, (int)(a->n_nodes + 1));
  p.cub_bytes = b1 > b2 ? b1 : b2;
  p.cub_bytes = p.cub_bytes > b3 ? p.cub_bytes : b3;
  p.cub_tmp = c.take<char>(p.cub_bytes);
}

static int validate_mass(const fm_mass_args *a, const char *who) {
  FM_REQUIRE(a != nullptr, FM_ERR_ARG, "%s: null args", who);
  FM_REQUIRE(a->n_elems >= 0 && a->n_nodes >= 0 && a->n_qpoints >= 0, FM_ERR_SHAPE, "%s: negative extent", who);
  FM_REQUIRE(a->nodes_per_elem >= 1 && a->nodes_per_elem <= kMaxNb, FM_ERR_SHAPE,
             "%s: nodes_per_elem=%d outside [1, %d]", who, a->nodes_per_elem, kMaxNb);
  FM_REQUIRE(a->n_nodes < (1LL << 31) - 2, FM_ERR_SHAPE, "%s: too many nodes", who);
  FM_REQUIRE(n_triplets(a) < (1LL << 31) - 2, FM_ERR_SHAPE, "%s: %lld triplets exceed the 2^31 limit", who,
             (long long)n_triplets(a));
  if (a->n_elems > 0) {
    FM_REQUIRE(a->elems && a->nodes && a->tabulated && (a->n_qpoints == 0 || a->qweights), FM_ERR_ARG,
               "%s: null input", who);
  }
  return FM_OK;
}

// One kernel per number of nodes of an element.
template <typename T, int NB>
static void mass_elements(const fm_mass_args *a, MassPlan &p, cudaStream_t st) {
  mass_local_kernel<T, NB><<<(unsigned)ceil_div(a->n_elems, 128), 128, 0, st>>>(
      a->n_elems, a->elems, a->n_nodes, static_cast<const T *>(a->nodes), a->n_qpoints,
      static_cast<const T *>(a->qweights), static_cast<const T *>(a->tabulated), static_cast<T *>(p.vals), p.degree,
      p.place, p.status + kMassBad, p.status + kMassOver);
  count_launch();
}
template <typename T, int NB>
static void mass_columns(const fm_mass_args *a, MassPlan &p, T *lump, cudaStream_t st) {
  const int64_t count = a->n_elems * NB;
  mass_around_kernel<NB><<<(unsigned)ceil_div(count, 256), 256, 0, st>>>(count, a->elems, a->n_nodes, p.start, p.place,
                                                                         p.around, p.status + kMassOver);
  count_launch();
  mass_columns_kernel<T, NB><<<(unsigned)ceil_div(a->n_nodes, kColWarps), 32 * kColWarps, 0, st>>>(
      a->n_nodes, a->elems, static_cast<const T *>(p.vals), p.start, p.around, p.rows, static_cast<T *>(p.data),
      p.colcount, lump, p.status + kMassOver);
  count_launch();
}
template <typename T>
static void mass_by_size(const fm_mass_args *a, MassPlan &p, bool columns, T *lump, cudaStream_t st) {
#define FM_MASS_CASE(NB) \
  case NB: return columns ? mass_columns<T, NB>(a, p, lump, st) : mass_elements<T, NB>(a, p, st);
  switch (a->nodes_per_elem) {
    FM_MASS_CASE(1) FM_MASS_CASE(2) FM_MASS_CASE(3) FM_MASS_CASE(4) FM_MASS_CASE(5)
    FM_MASS_CASE(6) FM_MASS_CASE(7) FM_MASS_CASE(8) FM_MASS_CASE(9) FM_MASS_CASE(10)
  }
#undef FM_MASS_CASE
}

static int mass_scan(MassPlan &p, const int *in, int *out, int64_t n, cudaStream_t st) {
  size_t cb = p.cub_bytes;
  FM_CUDA(cub::DeviceScan::ExclusiveSum(p.cub_tmp, cb, in, out, (int)n, st));
  count_launch();
  return FM_OK;
}

// Reads the status words and refuses a connectivity out of range.
static int mass_status(MassPlan &p, int64_t N, int (&h)[kMassWords], const char *who, cudaStream_t st) {
  FM_CUDA(cudaMemcpyAsync(h, p.status, sizeof(h), cudaMemcpyDeviceToHost, st));
  FM_CUDA(cudaStreamSynchronize(st));
  FM_REQUIRE(h[kMassBad] == 0, FM_ERR_SHAPE, "%s: element connectivity refers to a node outside [0, %lld)", who,
             (long long)N);
  return FM_OK;
}

// Builds the CSC of the assembled matrix: indptr in p.indptr, and rows and
// values in `indices` and `data` (capacity entries) when non-null; or, with
// `lump`, the sums of the columns.
//
// A cylinder of 60,000 nodes in tetrahedra, FP64 on a B200, kernel time of one
// build with a radix sort of all triplets against this: 720 us, 206 us (columns
// 138 us, element matrices 40 us).
template <typename T>
static int mass_build(fm_ctx *ctx, const fm_mass_args *a, MassPlan &p, int64_t *nnz_out, int32_t *indices, T *data,
                      int64_t capacity, T *lump, const char *who) {
  cudaStream_t st = ctx->stream;
  const int64_t K = n_triplets(a), N = a->n_nodes;
  const int nb = a->nodes_per_elem;
  int h[kMassWords] = {0, 0, 0, 0};
  FM_REQUIRE(K == 0 || N > 0, FM_ERR_SHAPE, "%s: element connectivity refers to a node outside [0, %lld)", who,
             (long long)N);
  FM_CUDA(cudaMemsetAsync(p.status, 0, kMassWords * sizeof(int), st));
  FM_CUDA(cudaMemsetAsync(p.degree, 0, (N + 2) * sizeof(int), st));
  FM_CUDA(cudaMemsetAsync(p.colcount, 0, (N + 2) * sizeof(int), st));
  if (K > 0) {
    mass_by_size<T>(a, p, false, nullptr, st);
    FM_TRY(check_launch("mass_local_kernel"));
    FM_TRY(mass_scan(p, p.degree, p.start, N + 1, st));
    mass_by_size<T>(a, p, true, lump, st);
    FM_TRY(check_launch("mass_columns_kernel"));
  }
  if (!lump) {
    FM_TRY(mass_scan(p, p.colcount, p.indptr, N + 1, st));
    FM_CUDA(cudaMemcpyAsync(p.status + kMassNnz, p.indptr + N, sizeof(int), cudaMemcpyDeviceToDevice, st));
  }
  FM_TRY(mass_status(p, N, h, who, st));
  if (h[kMassOver]) {
    // some column has more triplets than a warp orders: sort them all
    mass_triplets_kernel<<<(unsigned)ceil_div(K, 256), 256, 0, st>>>(K, nb, a->elems, p.keys_in, p.ord_in);
    count_launch();
    FM_TRY(check_launch("mass_triplets_kernel"));
    size_t cb = p.cub_bytes;
    FM_CUDA(cub::DeviceRadixSort::SortPairs(p.cub_tmp, cb, p.keys_in, p.keys_out, p.ord_in, p.ord_out, (int)K, 0, 64,
                                            st));
    count_launch();
    mass_heads_kernel<<<(unsigned)ceil_div(K, 256), 256, 0, st>>>(p.keys_out, K, p.head);
    count_launch();
    FM_TRY(check_launch("mass_heads_kernel"));
    cb = p.cub_bytes;
    FM_CUDA(cub::DeviceScan::InclusiveSum(p.cub_tmp, cb, p.head, p.uid, (int)K, st));
    count_launch();
    FM_CUDA(cudaMemcpyAsync(p.status + kMassNnz, p.uid + (K - 1), sizeof(int), cudaMemcpyDeviceToDevice, st));
    FM_TRY(mass_status(p, N, h, who, st));
  }
  const int64_t nnz = h[kMassNnz];
  if (nnz_out) *nnz_out = nnz;
  const bool write = data != nullptr;
  if (write) {
    FM_REQUIRE(capacity >= nnz, FM_ERR_NOMEM, "%s: output capacity %lld < nnz %lld", who, (long long)capacity,
               (long long)nnz);
  }
  if (h[kMassOver]) {
    T *to = lump ? static_cast<T *>(p.lump_data) : data;
    FM_CUDA(cudaMemsetAsync(p.colcount, 0, (N + 2) * sizeof(int), st));
    mass_collapse_kernel<T><<<(unsigned)ceil_div(K, 256), 256, 0, st>>>(
        p.keys_out, p.ord_out, static_cast<const T *>(p.vals), p.head, p.uid, K, indices, to, p.colcount,
        to != nullptr ? 1 : 0);
    count_launch();
    FM_TRY(check_launch("mass_collapse_kernel"));
    FM_TRY(mass_scan(p, p.colcount, p.indptr, N + 1, st));
    if (lump) {
      mass_lump_kernel<T><<<(unsigned)ceil_div(N, 256), 256, 0, st>>>(p.indptr, to, N, lump);
      count_launch();
      FM_TRY(check_launch("mass_lump_kernel"));
    }
  } else if (write && nnz > 0) {
    mass_pack_kernel<T><<<(unsigned)ceil_div(N * 16, 256), 256, 0, st>>>(
        N, nb, p.start, p.indptr, p.rows, static_cast<const T *>(p.data), indices, data);
    count_launch();
    FM_TRY(check_launch("mass_pack_kernel"));
  } else if (lump && K == 0) {
    FM_CUDA(cudaMemsetAsync(lump, 0, N * sizeof(T), st));
  }
  return FM_OK;
}

}  // namespace fm

using namespace fm;

extern "C" {

int fm_mass_workspace_size(const fm_mass_args *a, int is_double, size_t *bytes) {
  FM_REQUIRE(bytes != nullptr, FM_ERR_ARG, "fm_mass_workspace_size: null output");
  FM_TRY(validate_mass(a, "fm_mass_workspace_size"));
  Carve c(nullptr, 0);
  MassPlan p;
  carve_mass(c, a, is_double, p);
  *bytes = c.used;
  return FM_OK;
}

int fm_mass_assemble(fm_ctx *ctx, const fm_mass_args *a, int is_double, int64_t *nnz_out, int32_t *indptr,
                     int32_t *indices, void *data, int64_t capacity, void *workspace, size_t workspace_bytes) {
  FM_TRY(ctx_ok(ctx));
  FM_TRY(validate_mass(a, "fm_mass_assemble"));
  FM_REQUIRE(nnz_out != nullptr, FM_ERR_ARG, "fm_mass_assemble: null nnz_out");
  FM_REQUIRE((indices == nullptr) == (data == nullptr), FM_ERR_ARG,
             "fm_mass_assemble: indices and data must be given together");
  DeviceGuard g(ctx->device);
  Carve cv(workspace, workspace_bytes);
  MassPlan p;
  carve_mass(cv, a, is_double, p);
  FM_TRY(carve_ok(cv, "fm_mass_assemble"));
  int st;
  if (is_double)
    st = mass_build<double>(ctx, a, p, nnz_out, indices, static_cast<double *>(data), capacity, nullptr,
                            "fm_mass_assemble");
  else
    st = mass_build<float>(ctx, a, p, nnz_out, indices, static_cast<float *>(data), capacity, nullptr,
                           "fm_mass_assemble");
  FM_TRY(st);
  if (indptr) {
    FM_CUDA(cudaMemcpyAsync(indptr, p.indptr, (a->n_nodes + 1) * sizeof(int), cudaMemcpyDeviceToDevice,
                            ctx->stream));
  }
  return FM_OK;
}

int fm_mass_lumped(fm_ctx *ctx, const fm_mass_args *a, int is_double, void *out, void *workspace,
                   size_t workspace_bytes) {
  FM_TRY(ctx_ok(ctx));
  FM_TRY(validate_mass(a, "fm_mass_lumped"));
  FM_REQUIRE(out != nullptr || a->n_nodes == 0, FM_ERR_ARG, "fm_mass_lumped: null output");
  DeviceGuard g(ctx->device);
  Carve cv(workspace, workspace_bytes);
  MassPlan p;
  carve_mass(cv, a, is_double, p);
  FM_TRY(carve_ok(cv, "fm_mass_lumped"));
  if (a->n_nodes == 0) return FM_OK;
  if (is_double)
    return mass_build<double>(ctx, a, p, nullptr, nullptr, nullptr, 0, static_cast<double *>(out), "fm_mass_lumped");
  return mass_build<float>(ctx, a, p, nullptr, nullptr, nullptr, 0, static_cast<float *>(out), "fm_mass_lumped");
}

}  // extern "C"
