// Pieces shared by the Signal forms: the mass-weighted magnetisation M * Mxy,
// the distinct-time runs of the sample times, how far the samples factor, and
// the tile list that maps thread blocks to runs.
#pragma once
#include "motion.cuh"

namespace fm {

// Samples per tile of the plain (CUDA-core) forms.
constexpr int kPlainThreads = 256;

// CSR view of the sparse mass matrix, rows in Eigen's accumulation order.
struct Csr {
  int *rowptr;   // (rows + 1,)
  int *fill;     // (rows,)
  int *col;      // (nnz,)
  int *pos;      // (nnz,) position of the entry in the CSC arrays
  void *cub_tmp;
  size_t cub_bytes;
};

// Error bits recorded on the device during a Signal call.
constexpr int kErrTimeout = 1;      // a tensor-core pipeline wait ran out
constexpr int kErrSparseRow = 2;    // a row index of M outside [0, rows)
constexpr int kErrTableCalls = 4;   // TABLE motion entries != distinct-time runs
constexpr int kErrPhaseRange = 8;   // a tensor-core phase k . r or phi t may be out of its reduction's range

// Control words of one problem (zeroed when its descriptor is written).
constexpr int kCtlFlags = 0;    // kFlag* bits found over the samples and M
constexpr int kCtlRuns = 1;     // distinct-time runs
constexpr int kCtlFac = 2;      // factored runs
constexpr int kCtlTiles = 3;    // tiles of the other runs
constexpr int kCtlSplits = 4;   // node splits (tensor-core form)
constexpr int kCtlChunk = 5;    // nodes per split (tensor-core form)
constexpr int kCtlError = 6;    // kErr* bits
constexpr int kCtlPhi = 7;      // largest |phi| (float bits; a NaN counts as largest; tensor-core form)
constexpr int kCtlTime = 8;     // largest |t|, NaN apart (float bits; tensor-core form)
constexpr int kCtlOrder = 9;    // entries of the matrix's long rows put in order
constexpr int kCtlWords = 16;

// A slab is the Ls = lines x kz samples of one readout index.
constexpr int kFlagRuns = 1;           // some slab is not exactly one run
constexpr int kFlagSlabs = 2;          // some slab breaks k = kp + kq (checked additively in FP64)
constexpr int kFlagOffsets = 4;        // some slab's kz offsets differ from the first slab's
constexpr int kFlagNotDiagonal = 8;    // M has as many entries as rows but is not diagonal
constexpr int kFlagInSlab = 1 << 8;    // << c: component c of k varies inside some slab
constexpr int kFlagAcross = 1 << 11;   // << c: component c differs from the first slab's
constexpr int kFlagAlongKz = 1 << 14;  // << c: component c varies along some line's kz values
constexpr int kFlagOverLines = 1 << 17;  // << c: component c varies over some slab's lines at one kz

// Components of k that go with the run, and whether the samples factor as
// k(i, j, k) = k_run(i) + k_slab(j, k): every slab is one run and each component
// is either the same throughout every slab (it goes with the run) or the same
// in every slab (it goes with the place in the slab).
__device__ inline int prep_run_comps(const int *ctl) { return (ctl[kCtlFlags] / kFlagAcross) & 7; }
__device__ inline bool prep_static(const int *ctl) {
  const int f = ctl[kCtlFlags];
  return !(f & kFlagRuns) && ((f / kFlagInSlab) & (f / kFlagAcross) & 7) == 0;
}

// Descriptor of one problem's preparation, in device memory.
struct PrepDev {
  int64_t S, N, V;
  int Ls, n_lines, n_kz, n_ro;
  int n_chunks, chunk;   // the samples in n_chunks stretches of `chunk`
  int tile;              // samples per tile of an unfactored run
  int slab_cover;        // slabs that factor by components are not listed as tiles (CUDA-core forms)
  int run_cover;         // nor is anything where the runs factor out
  int stat;              // runs may factor out (no motion, several runs of several samples)
  int slabs;             // slabs may factor: factored runs are listed apart from the tiles
  int turns;             // the largest |phi| and |t| are wanted
  int diag;              // M holds as many entries as rows: diagonal unless shown otherwise
  int vgroup;            // columns per group of MM (0: one (N, V) matrix)
  int64_t table_calls;   // entries of a TABLE motion, -1 without one
  const void *kx, *ky, *kz, *t, *phi;
  const int *indptr, *indices;
  const void *data, *Mxy;
  void *MM;
  int *ctl;
  unsigned char *slab_bad;   // (n_ro,) slab is not one run or does not factor
  int *chunk_starts, *chunk_fac, *chunk_tiles;  // (n_chunks,) counts per stretch
  int *start;            // (S + 1,) run starts; start[n_runs] = S
  double *run_t;         // (S,) time of each run, widened to double
  int *frun;             // factored runs, ascending
  int2 *tiles;           // (run, first sample within it) of every other tile
  float *weights;        // (n_runs, slots) TERMS motion weights
  MotionDev md;
  Csr csr;
};

// Components of k that go with kz within a slab, and whether every run is a
// slab whose k factors as k_line(j) + k_kz(k), each component in one factor.
__device__ inline int prep_kz_comps(const int *ctl) { return (ctl[kCtlFlags] / kFlagAlongKz) & 7; }
__device__ inline bool prep_slab(const int *ctl) {
  const int f = ctl[kCtlFlags];
  return !(f & kFlagRuns) && ((f / kFlagAlongKz) & (f / kFlagOverLines) & 7) == 0;
}

// The CUDA-core form that sums a problem.  A problem whose motion table does not
// match its runs goes to the unfactored form, for which it has no tiles.
enum { kFormRuns, kFormSlabs, kFormPlain };
__device__ inline int prep_form(bool run_cover, bool slab_cover, const int *ctl) {
  if (ctl[kCtlError] & kErrTableCalls) return kFormPlain;
  return run_cover && prep_static(ctl) ? kFormRuns : (slab_cover && prep_slab(ctl) ? kFormSlabs : kFormPlain);
}

// Scratch of one problem: carved the same way when sizing and when running.
// `tensor_core`: factored slabs are listed for the tensor-core form (else for
// the factored CUDA-core form).
void carve_prep(Carve &c, const fm_signal_args *a, int tile, bool tensor_core, int vgroup, size_t real_bytes, int *ctl,
                PrepDev &p);
// Fills the rest of the descriptor from the arguments.
void fill_prep(const fm_signal_args *a, PrepDev &p);

// Queues the preparation of n problems (descriptors `host`, copied to the
// device array `dev`): runs, factoring, M * Mxy, motion weights and tiles.
// No host synchronisation and no copy from host memory.
template <typename T>
int launch_prep(const fm_signal_args *probs, const PrepDev *host, int n, PrepDev *dev, cudaStream_t st);

// Reads the error words of n problems (ctl: n rows of kCtlWords), waits for
// the stream and maps the first error to a status with a message.
int report_errors(const int *ctl, int n, cudaStream_t st, const char *who);

// Element of M Mxy for node n, column v: (N, V) rows, or per group of
// `vgroup` columns (N, ld) rows with ld = the group's columns rounded up to
// even (16-byte rows for the bulk copies), groups one after the other.
__host__ __device__ inline int64_t mm_index(int64_t n, int64_t v, int64_t N, int64_t V, int vgroup) {
  if (vgroup == 0) return n * V + v;
  const int64_t g = v / vgroup;
  const int64_t cols = (V - g * vgroup) < vgroup ? (V - g * vgroup) : vgroup;
  return g * N * vgroup + n * ((cols + 1) & ~(int64_t)1) + (v - g * vgroup);
}

}  // namespace fm
