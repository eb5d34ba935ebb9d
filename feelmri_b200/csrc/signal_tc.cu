// Split-BF16 tcgen05 tensor-core form of Signal.
//
// Same result as Signal<float> (cpp/feelmri/MRI.cpp:38-159 / :196-298): for
// each sample s of run g (time t_g, node positions r_n = r0_n + d_n(t_g))
//   K[s, v] = sum_n exp(-2 pi i k_s . r_n) * W_g[n, v],
//   W_g[n, v] = (M * Mxy)[n, v] * exp(-t_g / T2_n) * exp(i phi_n t_g),
// computed as a dense complex GEMM on the 5th-generation tensor cores:
//
// * Factoring.  A run whose samples form one complete Cartesian (line, kz)
//   slab with k(j, k) == kp_j + kq_k exactly (checked in FP64) is written as
//   C[p, (q, v)] = sum_n A[p, n] B[n, (q, v)] with A = exp(-2 pi i kp . r) and
//   B = exp(-2 pi i kq . r) W: P = lines rows, Q = kz values times V columns.
//   Every other run uses P = its samples and Q = 1 (B = W).
// * Real stacking.  Node n contributes two K entries: A'[p][2n..2n+1] =
//   (Re A, -Im A) and, in two blocks of B rows, B'^T[(q,v,re)][2n..] =
//   (Re B, Im B) and B'^T[(q,v,im)][2n..] = (Im B, -Re B), so column
//   (q,v,re) of C' is Re C and column (q,v,im) is Im C.
// * Split BF16.  Each operand x is stored as hi = bf16(x), lo = bf16(x - hi);
//   hi*hi + hi*lo + lo*hi accumulate in FP32 in tensor memory.
// * Phases.  k . r is evaluated in FP64 and reduced modulo one cycle (in
//   fixed point, to 2^-24 cycles) before the FP32 sin/cos, so far nodes at
//   high k keep their digits.
//
// Block (persistent, one per SM, 16 warps, each with a role of its own and
// mbarriers between them): warps 0-12 write the operand tiles into a ring of
// stages (16 nodes each) in shared memory, in the 64-byte swizzled K-major
// layout; warps 13 and 14 form the node blocks (128 nodes: moved positions,
// weights) ahead of them; one thread of warp 15 issues the MMAs of each written
// stage and releases its slot by tcgen05.commit.  The tensor core's FP32
// accumulation truncates, so the accumulator only collects 32 stages or fewer; warps 0-7
// then fold it into an FP32 (round-to-nearest) running sum kept in the other
// half of tensor memory.  Blocks loop over work units (row/column tile of a run
// x node range), each role on its own.  All waits are bounded: on timeout the
// block records an error, lets its MMAs finish and frees its tensor memory.
//
// What bounds it: operand writing, i.e. the instruction rate of the half-rate
// integer pipe and FP64 beside running MMAs; a stage takes about 1,600 cycles
// on wide tiles (128 pairs of 4 columns; its MMAs need 768), 900 on generic
// ones.  Measured on a B200, with one barrier for the whole block every two or
// four stages and one warp writing operands and issuing MMAs before:
// 200,740 nodes x 96 x 96 x 32 x 4 columns 9,274 -> 8,070 us, radial 50,021 x
// 65,536 x 8 columns with 10 modes 8,687 -> 5,200, 16 uneven phantoms 3,821 ->
// 2,470 (with runs as columns, kTcRuns).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "signal_common.cuh"
#include "tc_ptx.cuh"

namespace fm {

constexpr int kTcRows = 128;        // UMMA M
constexpr int kTcNodes = 16;        // nodes per stage -> K = 32 (two UMMA K steps)
constexpr int kTcMinRing = 3, kTcMaxRing = 8;  // pipeline stages in shared memory
constexpr int kTcBlockNodes = 128;  // nodes whose per-run data is formed together
constexpr int kTcStagesPerBlock = kTcBlockNodes / kTcNodes;
constexpr int kTcThreads = 512;
constexpr int kTcVGroup = 8;        // Mxy columns per launch
// Warp roles.  Warps 0-12 write the operand tiles, 13 and 14 form the node
// blocks, 15 issues the MMAs.  A stage's A is written by one warp per 32 rows,
// its B tile by one or two warps; such groups take the stages in turn, so that
// each warp waits, fences and signals once for all it does in a stage.  No
// more groups take turns than the ring has slots: a warp's next slot has then
// been released at most one round ago, and its barrier's parity is
// unambiguous.  Warps 0-7 also fold the accumulator and write the results.
constexpr int kTcDrainWarps = 8;
constexpr int kTcOperandWarps = 13;
constexpr int kTcStageArrivals = 6;  // at most 4 A and 2 B warps; the first A warp arrives for the missing ones
constexpr int kTcNodeWarp = 13;
constexpr int kTcMmaWarp = 15;
// Stages accumulated in the tensor-memory accumulator before it is folded
// into an FP32 round-to-nearest running sum (also in tensor memory).  The
// tensor core's FP32 accumulation truncates, so its error grows with the
// number of MMAs added into one accumulator; 32 stages (512 nodes, 192 MMAs)
// keep it near 1e-5.  On wide tiles all three products go to one accumulator, on
// narrow ones two (tensor memory below), and where runs are columns the turns
// (tc_runs_row) leave no element of the strongest samples 0: there 12 stages (72
// MMAs) keep the error at what such problems had as narrow or generic tiles.
// 198,606 nodes, 78 x 22 samples x 2 columns, on a B200: error 3.5e-6 with 32 stages,
// 2.1e-6 with 21, 1.3e-6 with 12 (1.4e-6 as generic tiles); uneven batch 1% slower
// than with 21.
constexpr int kTcDrain = 32, kTcDrainRuns = 12;
// Node buffers: one is written while others are still read.  The operand
// warps are up to a ring apart, so with two buffers of eight stages the next
// block was often late.
constexpr int kTcMinNodeBufs = 2, kTcMaxNodeBufs = 4;
constexpr uint64_t kTcWaitNs = 2000000000ull;
constexpr uint32_t kAStageBytes = kTcRows * 2 * kTcNodes * 2;  // 128 rows x 32 K x bf16 = 8 KB

// A work item: `rows` lines from line p0 and columns q0.. of run `run`, or
// (stacked problems) `rows` consecutive lines of the problem's runs laid end
// to end, from line p0 of run `run` on: unit row i is line (p0 + i) % P of
// run run + (p0 + i) / P (P lines per run), nrun runs in all, and every run
// shares the columns.  The runs then differ only in their times, so each
// run's decay and off-resonance factor D_r(n) = exp(-t_r / T2_n)
// exp(i phi_n t_r) moves into its A rows (A = exp(-2 pi i kp . r) D_r) and
// B = exp(-2 pi i kq . r) (M Mxy) is the same for all of them: the whole
// product is read.
struct TcItem {
  int run, p0, q0, nrun, rows;
};

// Kinds of launch entries (one problem's Mxy column group each).
constexpr int kTcSlab = 0;     // factored runs: rows lines, columns (kz, v)
constexpr int kTcGeneric = 1;  // other runs: rows samples, columns v
// Runs as columns, for a problem without motion whose k factors between the
// run and the place in the slab (prep_static): rows are the samples of a
// slab, columns (run, v); A = exp(-2 pi i k_slab . r), B = exp(-2 pi i k_run . r)
// exp(-t / T2) exp(i phi t) M Mxy, each node rotated by a turn of its own in A and
// back in B (tc_runs_row).  Slabs of few kz values then give wide
// tiles: a 32 x 32 x 8 grid of one coil has 64 units of 8 pairs as lines x kz
// (16 pairs of columns for 128 lines of 4 runs) and 2 units of 32 pairs here.
constexpr int kTcRuns = 2;
constexpr int kTcKinds = 3;

struct TcDev {
  int64_t N, S, V;
  int v0, VG;
  int n_lines, n_kz;
  const float *kx, *ky, *kz;
  const float *r0, *phi, *T2;
  const float2 *MM;
  MotionDev md;
  const float *weights;
  const float *table;
  const double *run_t;
  const int *start;   // run starts (PrepDev)
  const int *frun;    // factored runs
  const int2 *tiles;  // tiles of the generic runs
  int *ctl;           // control words of the problem
  int Qt, NT, kind;
  int drain;         // stages of an accumulation group
  int RU;            // lines per stacked unit
  int use_runs;      // runs become columns where k factors that way (kTcRuns)
  int prob, first, n_of, max_splits;  // the problem, its first entry and its entries
  int wrows;         // rows per node buffer: VG weight rows, then (stacked runs) nrun D rows
  int stacked;       // items may hold several runs (D in the A rows, B without decay)
  int mm_ld;         // row stride of MM (float2): this group's columns, padded to even
  int tma;           // node blocks are staged by bulk copies (aligned inputs, room in smem)
  int mstage;        // 3 r: a single POD term's mode rows are staged with each node block (0: read from global)
  float2 *partials; // (splits, S, V) when splits > 1
  float2 *out;
};

// Shared-memory layout of a launch, the same for all its entries (the warps
// cross from one unit to the next on their own, so a ring slot or node buffer
// must not move): barriers, `ring` stages, two to four node buffers (positions,
// weight rows), two staging areas of raw node blocks.
struct TcGeom {
  uint32_t stage_bytes, ring;
  uint32_t node_bufs, pos, w, wrows, raw, raw_bytes, total;
};

// One launch works through a table of entries (one per problem, Mxy column
// group and run kind); the device-side plan gives each entry's units.
struct TcBatchDev {
  const TcDev *entries;
  const int *offsets;  // device: n_entries + 1 running unit counts
  int n_entries;
  TcGeom geom;
};

// Work list of one entry, from the problem's control words.
struct TcWork {
  int splits, n_items;
  bool stack;  // items are consecutive lines of the runs laid end to end
  int64_t chunk;
  float2 *out;
};

// Runs can be stacked into one unit when the positions do not depend on the
// run (no motion) and every run is a factored slab of the full (lines x kz)
// shape with the same kz offsets, exactly (flags of the sample scan).
__device__ inline bool tc_stacked(const TcDev &p) {
  return p.stacked && !(p.ctl[kCtlFlags] & (kFlagRuns | kFlagSlabs | kFlagOffsets));
}

__device__ inline int tc_items_per_run(const TcDev &p) {
  return (int)(ceil_div(p.n_lines, kTcRows) * ceil_div(p.n_kz, p.Qt));
}

__device__ inline int tc_n_items(const TcDev &p) {
  if (p.use_runs && prep_static(p.ctl)) {
    if (p.kind != kTcRuns) return 0;
    return (int)(ceil_div((int64_t)p.n_lines * p.n_kz, kTcRows) * ceil_div(p.ctl[kCtlRuns], p.Qt));
  }
  if (p.kind == kTcRuns) return 0;
  if (p.kind == kTcGeneric) return p.ctl[kCtlTiles];
  if (tc_stacked(p)) return (int)ceil_div((int64_t)p.ctl[kCtlRuns] * p.n_lines, (int64_t)p.RU);
  return p.ctl[kCtlFac] * tc_items_per_run(p);
}

__device__ inline TcWork tc_work(const TcDev &p) {
  TcWork W;
  W.splits = p.ctl[kCtlSplits];
  W.chunk = p.ctl[kCtlChunk];
  W.n_items = tc_n_items(p);
  W.stack = p.kind == kTcSlab && tc_stacked(p);
  W.out = W.splits > 1 ? p.partials : p.out;
  return W;
}

__device__ inline TcItem tc_item(const TcDev &p, const TcWork &W, int i) {
  TcItem t;
  if (p.kind == kTcGeneric) {
    const int2 k = p.tiles[i];
    t.run = k.x; t.p0 = k.y; t.q0 = 0; t.nrun = 1;
    t.rows = min(kTcRows, p.start[k.x + 1] - p.start[k.x] - k.y);
  } else if (p.kind == kTcRuns) {
    const int nq = (int)ceil_div(p.ctl[kCtlRuns], p.Qt);
    t.run = 0; t.nrun = 1;
    t.p0 = (i / nq) * kTcRows;
    t.q0 = (i % nq) * p.Qt;
    t.rows = min(kTcRows, p.n_lines * p.n_kz - t.p0);
  } else if (W.stack) {
    const int64_t L0 = (int64_t)i * p.RU, total = (int64_t)p.ctl[kCtlRuns] * p.n_lines;
    t.run = (int)(L0 / p.n_lines);
    t.p0 = (int)(L0 - (int64_t)t.run * p.n_lines);
    t.q0 = 0;
    t.rows = (int)min((int64_t)p.RU, total - L0);
    t.nrun = (t.p0 + t.rows - 1) / p.n_lines + 1;
  } else {
    const int c = tc_items_per_run(p), nq = (int)ceil_div(p.n_kz, p.Qt);
    const int w = i % c;
    t.run = p.frun[i / c];
    t.p0 = (w / nq) * kTcRows;
    t.q0 = (w % nq) * p.Qt;
    t.nrun = 1;
    t.rows = min(kTcRows, p.n_lines - t.p0);
  }
  return t;
}

// A weight row of a node buffer is a row of real parts and one of imaginary
// parts, kWStride floats each (padded, so that 16-byte reads of different
// rows fall in different banks).
constexpr int kWStride = kTcBlockNodes + 4;
constexpr uint32_t kTcPosBytes = 4 * kTcBlockNodes * 8;  // x, y, z rows of a node buffer and one more (FP64)
constexpr int kTcComps = 4;  // x, y, z and (runs as columns) the run's time
constexpr uint32_t kTcSmemMax = 232448;  // dynamic shared memory a block may opt in to

// Barriers, the tensor-memory address and small shared values.
constexpr uint32_t kTcFront = 1024;
constexpr uint32_t kTcMisc = 256;
struct TcBars {
  uint64_t full[kTcMaxRing], empty[kTcMaxRing];
  uint64_t accfull, accfree;
  uint64_t nodefull[kTcMaxNodeBufs], nodeempty[kTcMaxNodeBufs], rawfull[2];
  uint64_t done;
};
static_assert(kTcMinRing >= 3, "three groups of A warps take turns");
static_assert(sizeof(TcBars) <= kTcMisc, "barriers fit before the other shared values");
struct TcMisc {
  uint32_t tmem;
  int abort_flag;
  int rmax[kTcMaxNodeBufs];  // largest |x| + |y| + |z| of each node buffer (float bits)
};

// Narrow and wide tiles (tensor-memory layout and MMAs below).
__host__ __device__ inline bool tc_narrow(int NT) { return NT <= 128; }

__host__ __device__ inline uint32_t tc_stage_bytes(int NT) { return 2 * kAStageBytes + 2 * NT * 2 * kTcNodes * 2; }

// Bytes of one raw node block: positions, T2, phi and the group's M Mxy rows.
__host__ __device__ inline uint32_t tc_raw_bytes(int mm_ld) {
  return kTcBlockNodes * (12 + 4 + 4 + 8 * mm_ld);
}

// Bytes of one node block's POD mode rows ([128][3 r] floats), staged after
// the raw block when TcDev::mstage (= 3 r) is set.
__host__ __device__ inline uint32_t tc_mode_bytes(int mstage) { return kTcBlockNodes * 4 * (uint32_t)mstage; }

// Byte offset of element (row, k) of a K-major operand tile with 32 K
// elements (64-byte rows) in the 64-byte swizzled layout: row r at r * 64,
// its 16-byte chunk c (elements 8c .. 8c + 7) stored at chunk position
// c ^ ((r >> 1) & 3), i.e. address bits 4-5 XOR bits 7-8.  Tiles start on
// 512-byte boundaries (8-row groups, SBO = 512), so the swizzle of a byte
// offset is the swizzle of its shared-memory address.  The tensor core reads
// this layout at full shared-memory bandwidth; the unswizzled layout's
// 16-byte core-matrix rows cap its operand reads, which dominates narrow
// (small N) MMAs.
__host__ __device__ inline uint32_t sw64_offset(uint32_t row, uint32_t k) {
  return row * 64 + ((((k >> 3) ^ (row >> 1)) & 3) << 4) + (k & 7) * 2;
}

// Two FP32 values in one 64-bit register pair: the packed add, multiply and
// multiply-add issue once for both.
struct F2 {
  unsigned long long v;
};
__device__ inline F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ inline void f2_get(F2 x, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ inline F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ inline F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

__device__ inline uint32_t bf16_pair(float a, float b) {
  uint32_t r;  // a in the low half (cvt.rn.bf16x2 puts its first source in the upper half)
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

// a - h and b - h' for the BF16 pair (h, h'), exactly: the mixed-precision
// multiply-add takes the BF16 operand as it is.  Shifting it into place first
// (two instructions of the half-rate integer pipe a pair) made a split twice
// as long: 8 cycles against 4.2.
__device__ inline void minus_bf16(float a, float b, uint32_t pair, float &da, float &db) {
  const uint16_t minus_one = 0xbf80;
  asm("{\n\t.reg .b16 l, h;\n\t"
      "mov.b32 {l, h}, %2;\n\t"
      "fma.rn.f32.bf16 %0, l, %3, %4;\n\t"
      "fma.rn.f32.bf16 %1, h, %3, %5;\n\t}"
      : "=&f"(da), "=f"(db)
      : "r"(pair), "h"(minus_one), "f"(a), "f"(b));
}

// hi = bf16(x), lo = bf16(x - hi) for the pair (a, b); bits of (hi_a, hi_b)
// and (lo_a, lo_b) with a in the low half.
__device__ inline void split_pair(float a, float b, uint32_t &hi, uint32_t &lo) {
  float la, lb;
  hi = bf16_pair(a, b);
  minus_bf16(a, b, hi, la, lb);
  lo = bf16_pair(la, lb);
}
// The same for (a, b) and for (b, -a).
__device__ inline void split_pair_im(float a, float b, uint32_t &hi, uint32_t &lo, uint32_t &hi_im, uint32_t &lo_im) {
  hi = bf16_pair(a, b);
  hi_im = bf16_pair(b, -a);
  float la, lb;
  minus_bf16(a, b, hi, la, lb);
  lo = bf16_pair(la, lb);
  lo_im = bf16_pair(lb, -la);
}

// cos and sin of 2 pi c for c in cycles given in FP64.  c is reduced modulo
// one in fixed point: adding 1.5 * 2^29 leaves a double whose last place is
// 2^-23, so its low 32 bits hold round(c * 2^23) modulo 2^32 and their low
// 23 bits, moved to the top of the word, are c - rint(c) in units of 2^-32
// (error at most 2^-24 cycles, for |c| < 2^28).  This keeps the reduction off
// the transcendental unit (no rint, no double-to-float conversion): one FP64
// add, a shift and an integer-to-float conversion, then the FP32 sin/cos.
// FP64 shares its unit with the tensor core (a DFMA takes 3.2 times as long
// while N = 256 MMAs run); forming the phases by 32 x 32-bit integer multiplies
// instead was slower all the same (flow case 9.6 against 8.3 ms), since the
// half-rate integer pipe is the busier one here.
__device__ inline void cycles_cos_sin(double c, float &co, float &s) {
  const int frac = (int)((unsigned)__double2loint(__dadd_rn(c, 805306368.0)) << 9);
  __sincosf(__int2float_rn(frac) * 1.4629180792671596e-09f, &s, &co);  // 2 pi / 2^32
}

__device__ inline void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  // no memory clobber: the stores are ordered before the proxy fence (also
  // volatile) that publishes them, and no generic load reads them back
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d));
}

__device__ inline void st_shared(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v));
}

struct TcUnit {
  TcItem it;
  int start;      // first sample of the first run
  int P;          // lines per run (factored) or samples of the run
  int split, Q_tile, n_stages, n_groups;
  int drain;      // TcDev::drain
  int rows;       // active A rows
  int64_t n_begin, n_end;
};

__device__ inline TcUnit tc_unit(const TcDev &p, const TcWork &W, int u) {
  TcUnit U;
  const int item = u % W.n_items;
  U.split = u / W.n_items;
  U.it = tc_item(p, W, item);
  U.start = p.start[U.it.run];
  U.P = p.kind == kTcSlab ? p.n_lines : p.start[U.it.run + 1] - U.start;
  U.Q_tile = p.kind == kTcSlab ? min(p.Qt, p.n_kz - U.it.q0)
                               : (p.kind == kTcRuns ? min(p.Qt, p.ctl[kCtlRuns] - U.it.q0) : 1);
  U.rows = U.it.rows;
  U.n_begin = (int64_t)U.split * W.chunk;
  U.n_end = min(p.N, U.n_begin + W.chunk);
  U.n_stages = U.n_end > U.n_begin ? (int)ceil_div(U.n_end - U.n_begin, kTcNodes) : 0;
  U.drain = p.drain;
  U.n_groups = (U.n_stages + U.drain - 1) / U.drain;
  return U;
}

// Entry of unit u: offsets[e] <= u < offsets[e + 1].
__device__ inline int tc_entry_of(const TcBatchDev &B, int u) {
  int lo = 0, hi = B.n_entries;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (B.offsets[mid] <= u) lo = mid; else hi = mid;
  }
  return lo;
}

// Run (relative to the unit's first) and line of unit row `row` (TcItem).
__device__ inline void tc_row_line(const TcDev &p, const TcUnit &U, int row, int &r, int &line) {
  if (p.stacked) {
    const int lr = U.it.p0 + row;
    r = lr / U.P;
    line = lr % U.P;
  } else {
    r = 0;
    line = U.it.p0 + row;
  }
}

// Output sample of unit row `row` and its first column, and the step from one
// column q to the next (every run of a stacked unit shares the columns).
__device__ inline void tc_out_sample(const TcDev &p, const TcUnit &U, int row, int64_t &s_row, int64_t &s_q) {
  int r, line;
  tc_row_line(p, U, row, r, line);
  if (p.kind == kTcRuns) {
    s_q = (int64_t)p.n_lines * p.n_kz;
    s_row = U.it.q0 * s_q + line;
    return;
  }
  s_q = 1;
  s_row = p.start[U.it.run + r] + (p.kind == kTcSlab ? (int64_t)line * p.n_kz + U.it.q0 : line);
}

// Bounded wait; false when it ran out, and at once after any earlier one of the
// block did (the flag lives in shared memory).  The MMA and node roles end with a
// failed wait; the operand warps, which share a barrier, walk on without waiting
// to the end of their unit and leave there together.  So a block ends soon after
// the first wait that ran out, whatever work is left.  Every arrival but the copies'
// is a single one: arrivals that no wait made room for then complete phases that
// nobody trusts any more, where a count above what a phase has left would fault.
__device__ inline bool tc_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  if (ptx::mbar_test_wait(bar, parity)) return true;
  if (*abort_flag) return false;
  if (ptx::mbar_wait(bar, parity, kTcWaitNs)) return true;
  *abort_flag = 1;
  return false;
}

// Ring position of a warp: slot and the parity its `full` barrier completes
// with (its `empty` barrier is waited for with the opposite one).
struct TcRing {
  uint32_t slot, phase;
  __device__ inline void seek(uint32_t stage, uint32_t ring) {
    slot = stage % ring;
    phase = (stage / ring) & 1;
  }
  __device__ inline void advance(uint32_t stages, uint32_t ring) {
    slot += stages;
    while (slot >= ring) {
      slot -= ring;
      phase ^= 1;
    }
  }
};

// float bits of |x| + |y| + |z| (a NaN compares above every number)
__device__ inline int tc_abs_sum(double x, double y, double z) {
  return __float_as_int((float)(fabs(x) + fabs(y) + fabs(z))) & 0x7fffffff;
}

// Rows of a node buffer where runs are columns: the components of k that go with the
// run come first, for B, which reads rows 0 to 2; A reads rows 1 to 3, the last of
// which is a turn of each node's own, in cycles, by which A is rotated and the
// weights back.  A is a function of the place alone there, so nodes in line have the
// same A, and with it the same error of its split; the errors of a line then add up
// to that of its whole sum.  With a turn of its own each node's error is another.
// 196,955 nodes of a grid, 105 x 105 x 16 samples, on a B200: error 1.24e-5 without
// turns, 7.6e-6 with them (8.3e-6 as lines x kz, whose A holds the nodes' decay).
// Where no component goes with the run, A takes all three and there is no turn.
__device__ inline int tc_runs_row(int cmask, int c) {
  const int in = __popc(cmask & ((1 << c) - 1));  // components before c that go with the run
  if (cmask == 0) return c + 1;
  return (cmask >> c) & 1 ? in : __popc(cmask) + c - in;
}

// A turn for node n in [0, 1): the bits of n well mixed.
__device__ inline double tc_node_turn(int64_t n) {
  uint32_t h = (uint32_t)n * 0x9e3779b1u;
  h = (h ^ (h >> 15)) * 0x85ebca77u;
  h ^= h >> 13;
  return (double)h * 0x1p-32;
}

// ---- node blocks ---------------------------------------------------------

// Raw data of one node block in a staging area.
struct TcRawView {
  const float *r0, *T2, *phi;
  const float2 *MM;
  const float *modes;
};
__device__ inline TcRawView tc_raw_view(const unsigned char *staging, int mm_ld) {
  TcRawView v;
  v.r0 = reinterpret_cast<const float *>(staging);
  v.T2 = v.r0 + 3 * kTcBlockNodes;
  v.phi = v.T2 + kTcBlockNodes;
  v.MM = reinterpret_cast<const float2 *>(v.phi + kTcBlockNodes);
  v.modes = reinterpret_cast<const float *>(staging + tc_raw_bytes(mm_ld));
  return v;
}

// What the node warps need of an entry and a unit, held in registers: reading
// the entry again for every node cost more than the nodes' arithmetic (a block
// took 5,100 cycles at 8 columns and 10 modes, 2,900 at 4 columns and one
// mode, and set the pace of the whole block).
struct TcNodeArgs {
  const float *r0, *T2, *phi, *modes, *wrun, *table;
  const float2 *MM;
  int VG, mm_ld, mstage, wrows, nrun;
  bool stacked, runs, turns;
  int row[3];  // rows of x, y, z in the node buffer
  float t;  // the run's time; stacked: lane k holds run k's
  float w;  // lane k: motion weight k of a staged term
};

__device__ inline TcNodeArgs tc_node_args(const TcDev &p, const TcUnit &U, int lane) {
  TcNodeArgs a;
  a.r0 = p.r0; a.T2 = p.T2; a.phi = p.phi;
  a.MM = p.MM;
  a.VG = p.VG; a.mm_ld = p.mm_ld; a.mstage = p.mstage; a.wrows = p.wrows; a.nrun = U.it.nrun;
  a.modes = p.mstage ? p.md.terms[0].modes : nullptr;
  a.wrun = p.weights ? p.weights + (int64_t)U.it.run * p.md.slots : nullptr;
  a.table = p.table ? p.table + (int64_t)U.it.run * p.N * 3 : nullptr;
  a.stacked = p.stacked != 0;
  a.runs = p.kind == kTcRuns;
  const int cmask = a.runs ? prep_run_comps(p.ctl) : 0;
  a.turns = cmask != 0;
  for (int c = 0; c < 3; ++c) a.row[c] = a.runs ? tc_runs_row(cmask, c) : c;
  a.t = (float)p.run_t[U.it.run + (a.stacked && lane < a.nrun ? lane : 0)];
  a.w = p.mstage && 3 * lane < p.mstage ? a.wrun[p.md.slot0[0] + lane] : 0.f;
  return a;
}

// Requests the raw data of the full node block at n0 (one thread).
__device__ inline void tc_request_block(const TcNodeArgs &a, int64_t n0, unsigned char *staging, uint64_t *rawfull) {
  const TcRawView v = tc_raw_view(staging, a.mm_ld);
  // the staging area's previous readers are past a barrier; order their
  // reads before the copies
  ptx::fence_proxy_async_smem();
  ptx::mbar_arrive_expect_tx(rawfull, tc_raw_bytes(a.mm_ld) + tc_mode_bytes(a.mstage));
  ptx::bulk_copy_g2s((void *)v.r0, a.r0 + 3 * n0, 12 * kTcBlockNodes, rawfull);
  ptx::bulk_copy_g2s((void *)v.T2, a.T2 + n0, 4 * kTcBlockNodes, rawfull);
  ptx::bulk_copy_g2s((void *)v.phi, a.phi + n0, 4 * kTcBlockNodes, rawfull);
  ptx::bulk_copy_g2s((void *)v.MM, a.MM + n0 * a.mm_ld, 8 * kTcBlockNodes * a.mm_ld, rawfull);
  // mode rows of node n0 onwards: 12 r bytes per node, n0 a multiple of 16
  // and the rows 16-byte aligned (checked on the host)
  if (a.mstage) ptx::bulk_copy_g2s((void *)v.modes, a.modes + n0 * a.mstage, tc_mode_bytes(a.mstage), rawfull);
}

// motion_disp's sum over the modes of a POD term in W modes a load.  A warp's
// nodes are rows apart, so each load is 32 requests whatever its width, and the two
// node warps must keep the pace that the whole block once set: 20,011 nodes x 64 x 64
// samples on a B200, 20 modes 676 us with single reads, 410 us; 64 modes 2029 us,
// 785 us (with nodes formed by four warps it was 620 us and 1633 us).
template <int W>
__device__ __forceinline__ void tc_pod_sum(const float *Phi, const float *wk, int r, float &tx, float &ty, float &tz) {
  using V = typename std::conditional<W == 4, float4, typename std::conditional<W == 2, float2, float>::type>::type;
  tx = 0.f; ty = 0.f; tz = 0.f;
#pragma unroll 2  // (what the kernel's registers take best)
  for (int m = 0; m < r; m += W) {
    const V a = __ldg(reinterpret_cast<const V *>(Phi + m)), b = __ldg(reinterpret_cast<const V *>(Phi + r + m)),
            c = __ldg(reinterpret_cast<const V *>(Phi + 2 * r + m));
    const float *pa = reinterpret_cast<const float *>(&a), *pb = reinterpret_cast<const float *>(&b),
                *pc = reinterpret_cast<const float *>(&c);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const float wm = wk[m + i];
      tx = fmaf(pa[i], wm, tx);
      ty = fmaf(pb[i], wm, ty);
      tz = fmaf(pc[i], wm, tz);
    }
  }
}

// motion_disp, the modes of each POD term read as wide as its rows are aligned.
__device__ __forceinline__ void tc_motion_disp(const MotionDev &md, const float *w, int64_t n, float &dx, float &dy,
                                               float &dz) {
  float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll 1
  for (int k = 0; k < md.n_terms; ++k) {
    const fm_motion_term &T = md.terms[k];
    const float *wk = w + md.slot0[k];
    float tx, ty, tz;
    if (T.kind == FM_TERM_RESPIRATORY) {
      tx = __fmul_rn(wk[0], T.direction[0]);
      ty = __fmul_rn(wk[0], T.direction[1]);
      tz = __fmul_rn(wk[0], T.direction[2]);
    } else {
      const int r = T.n_modes;
      const float *Phi = T.modes + (size_t)n * 3 * r;
      const unsigned by = (unsigned)(uintptr_t)T.modes | 4u * r;  // rows start, and components lie, at multiples of it
      if (by % 16 == 0) tc_pod_sum<4>(Phi, wk, r, tx, ty, tz);
      else if (by % 8 == 0) tc_pod_sum<2>(Phi, wk, r, tx, ty, tz);
      else tc_pod_sum<1>(Phi, wk, r, tx, ty, tz);
    }
    if (k == 0) { sx = tx; sy = ty; sz = tz; }
    else { sx = __fadd_rn(sx, tx); sy = __fadd_rn(sy, ty); sz = __fadd_rn(sz, tz); }
  }
  dx = sx; dy = sy; dz = sz;
}

// Node quantities of the block at n0 into a node buffer (one warp, nodes lane,
// lane + 32 ..): moved position (in FP64 for the phase
// products) and the decayed, off-resonance rotated weights
// W' = (M Mxy)[n, v] exp(-t / T2) exp(i phi t) of the run.  Nodes past the
// range get position 0 and zero weights, so they add nothing.  Returns the
// largest |x| + |y| + |z| for the phase range check (float bits).
__device__ __forceinline__ int tc_derive(const TcDev &p, const TcNodeArgs &a, int64_t n0, int64_t n_end, bool staged,
                                         const TcRawView &raw, unsigned char *buf, float *wblk, int slot0) {
  constexpr int kPer = kTcBlockNodes / 32, kStep = 32;
  double *pos = reinterpret_cast<double *>(buf);
  bool in[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) in[i] = n0 + slot0 + i * kStep < n_end;
  auto place = [&](int slot, bool inside, float &x, float &y, float &z) {
    if (staged) {
      x = raw.r0[3 * slot]; y = raw.r0[3 * slot + 1]; z = raw.r0[3 * slot + 2];
    } else if (inside) {
      const float *r = a.r0 + 3 * (n0 + slot);
      x = r[0]; y = r[1]; z = r[2];
    } else {
      x = y = z = 0.f;
    }
  };
  int rmax = 0;
  auto put_place = [&](int slot, float x, float y, float z) {
    pos[a.row[0] * kTcBlockNodes + slot] = (double)x;
    pos[a.row[1] * kTcBlockNodes + slot] = (double)y;
    pos[a.row[2] * kTcBlockNodes + slot] = (double)z;
    rmax = max(rmax, __float_as_int(fabsf(x) + fabsf(y) + fabsf(z)) & 0x7fffffff);
  };
  if (staged && a.mstage) {
    // the single POD term's sum (motion_disp's products in its order), the
    // mode rows read from the staged block
    const int rk = a.mstage / 3;
    float dx[kPer], dy[kPer], dz[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) dx[i] = dy[i] = dz[i] = 0.f;
#pragma unroll 2
    for (int k = 0; k < rk; ++k) {
      const float wm = __shfl_sync(0xffffffffu, a.w, k);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const float *Phi = raw.modes + (slot0 + i * kStep) * a.mstage + k;
        dx[i] = fmaf(Phi[0], wm, dx[i]);
        dy[i] = fmaf(Phi[rk], wm, dy[i]);
        dz[i] = fmaf(Phi[2 * rk], wm, dz[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      float x, y, z;
      place(slot0 + i * kStep, true, x, y, z);
      put_place(slot0 + i * kStep, x + dx[i], y + dy[i], z + dz[i]);
    }
  } else if (a.wrun || a.table) {
#pragma unroll 1
    for (int slot = slot0; slot < kTcBlockNodes; slot += kStep) {
      const int64_t n = n0 + slot;
      float x, y, z;
      place(slot, n < n_end, x, y, z);
      if (n < n_end) {
        float dx, dy, dz;
        if (a.wrun) {
          tc_motion_disp(p.md, a.wrun, n, dx, dy, dz);
        } else {
          dx = a.table[3 * n]; dy = a.table[3 * n + 1]; dz = a.table[3 * n + 2];
        }
        x = x + dx; y = y + dy; z = z + dz;
      }
      put_place(slot, x, y, z);
    }
  } else {
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      float x, y, z;
      place(slot0 + i * kStep, in[i], x, y, z);
      put_place(slot0 + i * kStep, x, y, z);
    }
  }
  float t2[kPer], phi[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int slot = slot0 + i * kStep;
    t2[i] = staged ? raw.T2[slot] : (in[i] ? a.T2[n0 + slot] : 1.f);
    phi[i] = staged ? raw.phi[slot] : (in[i] ? a.phi[n0 + slot] : 0.f);
  }
  // decay exp(-t / T2) and off-resonance rotation exp(i phi t) of a run: the
  // fast exponential of -t (1 / T2), and the phase phi t reduced in cycles in
  // FP64 before the fast sin/cos (cycles_cos_sin), as the A and B tiles do
  // (both within a few 1e-7 of the accurate functions).  Stacked: the weights
  // without decay (B), then one D_r = decay e^{i phi t_r} row per run (A).
  // Runs as columns: the weights without decay, rotated by the node's turn, then
  // 1 / T2 and (FP64) phi in cycles, from which B forms each run's factor.
  const int nd = a.runs ? 0 : (a.stacked ? a.nrun : 1);
  float inv_t2[kPer], er[kPer], ei[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) inv_t2[i] = __frcp_rn(t2[i]);
  if (a.runs) {
    double *ph = reinterpret_cast<double *>(wblk + 2 * (a.VG + 1) * kWStride);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int slot = slot0 + i * kStep;
      wblk[2 * a.VG * kWStride + slot] = in[i] ? inv_t2[i] : 0.f;
      ph[slot] = (double)phi[i] * 0.15915494309189535;
      const double turn = a.turns ? tc_node_turn(n0 + slot) : 0.0;
      pos[(a.turns ? 3 : 0) * kTcBlockNodes + slot] = turn;
      cycles_cos_sin(turn, er[i], ei[i]);  // A = exp(-2 pi i (k . r + turn))
    }
  }
#pragma unroll 1
  for (int k = 0; k < nd; ++k) {
    const float tg = a.stacked ? __shfl_sync(0xffffffffu, a.t, k) : a.t;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const float decay = in[i] ? __expf(-tg * inv_t2[i]) : 0.f;
      float so, co;
      cycles_cos_sin((double)(phi[i] * tg) * 0.15915494309189535, co, so);
      er[i] = in[i] ? decay * co : 0.f;
      ei[i] = in[i] ? decay * so : 0.f;
      if (a.stacked) {
        wblk[2 * (a.VG + k) * kWStride + slot0 + i * kStep] = er[i];
        wblk[(2 * (a.VG + k) + 1) * kWStride + slot0 + i * kStep] = ei[i];
      }
    }
  }
  const bool plain = a.stacked;
  auto put = [&](int v, int slot, float2 m, float dr, float di) {
    wblk[2 * v * kWStride + slot] = plain ? m.x : m.x * dr - m.y * di;
    wblk[(2 * v + 1) * kWStride + slot] = plain ? m.y : m.x * di + m.y * dr;
  };
#pragma unroll 1
  for (int v = 0; v < a.VG; v += 2) {  // rows of M Mxy hold column pairs
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int slot = slot0 + i * kStep;
      float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
      if (staged) m = *reinterpret_cast<const float4 *>(raw.MM + slot * a.mm_ld + v);
      else if (in[i]) m = *reinterpret_cast<const float4 *>(a.MM + (n0 + slot) * a.mm_ld + v);
      put(v, slot, make_float2(m.x, m.y), er[i], ei[i]);
      if (v + 1 < a.VG) put(v + 1, slot, make_float2(m.z, m.w), er[i], ei[i]);
    }
  }
  return rmax;
}

// ---- operand tiles -------------------------------------------------------

// Phases k . r of two nodes, in cycles; kRuns: less phi t (ph in cycles, time k[3]).
template <bool kRuns>
__device__ __forceinline__ void tc_phase2(const double *pos, const double (&k)[kTcComps], const double *ph, float &c0,
                                          float &s0, float &c1, float &s1) {
  const double2 x = *reinterpret_cast<const double2 *>(pos);
  const double2 y = *reinterpret_cast<const double2 *>(pos + kTcBlockNodes);
  const double2 z = *reinterpret_cast<const double2 *>(pos + 2 * kTcBlockNodes);
  double a = k[0] * x.x, b = k[0] * x.y;
  if (kRuns) {
    const double2 f = *reinterpret_cast<const double2 *>(ph);
    a = fma(-k[3], f.x, a);
    b = fma(-k[3], f.y, b);
  }
  cycles_cos_sin(fma(k[2], z.x, fma(k[1], y.x, a)), c0, s0);
  cycles_cos_sin(fma(k[2], z.y, fma(k[1], y.y, b)), c1, s1);
}

// A'[row][2n..2n+1] = (Re A, -Im A) = (cos, sin) of 2 pi kp . r_n of 8 nodes;
// in a stacked unit A is multiplied by the row's run factor D_r(n):
// (Re, -Im) of (cos - i sin)(dr + i di) = (cos dr + sin di, sin dr - cos di).
// addr: the row's first 16-byte chunk (hi tile); the second is d_k2 = +/-16
// bytes from it (swizzled chunk positions 2 half and 2 half + 1 differ in
// their lowest bit), the lo tile kAStageBytes on.
template <bool kStacked>
__device__ __forceinline__ void tc_write_a(const double *pos, const double (&kd)[kTcComps], const float *dp,
                                           uint32_t addr, int d_k2) {
  uint32_t h[8], l[8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    float c0, s0, c1, s1;
    tc_phase2<false>(pos + i, kd, nullptr, c0, s0, c1, s1);
    if (kStacked) {
      const float2 dr = *reinterpret_cast<const float2 *>(dp + i);
      const float2 di = *reinterpret_cast<const float2 *>(dp + kWStride + i);
      const float r0 = fmaf(c0, dr.x, s0 * di.x), r1 = fmaf(c1, dr.y, s1 * di.y);
      s0 = fmaf(s0, dr.x, -(c0 * di.x));
      s1 = fmaf(s1, dr.y, -(c1 * di.y));
      c0 = r0;
      c1 = r1;
    }
    split_pair(c0, s0, h[i], l[i]);
    split_pair(c1, s1, h[i + 1], l[i + 1]);
  }
  st_shared_v4(addr, h[0], h[1], h[2], h[3]);
  st_shared_v4(addr + d_k2, h[4], h[5], h[6], h[7]);
  st_shared_v4(addr + kAStageBytes, l[0], l[1], l[2], l[3]);
  st_shared_v4(addr + kAStageBytes + d_k2, l[4], l[5], l[6], l[7]);
}

// B'^T rows of one kz value q and 8 nodes, all VG columns: re row `row` =
// (Re B, Im B), im row NT/2 + row = (Im B, -Re B), B = e_q(n) W'(n, v),
// e_q = exp(-2 pi i kq . r_n), row = v Qt + q (the lanes of a warp hold
// consecutive q, so their 16-byte stores fall in different banks; rows
// q VG + v took 570 cycles a task at VG = 4 against 220).  wblk: the
// block's weight rows; node0: the first of the 8 nodes.
// kRuns: q is a run of time t and B also carries its decay and off-resonance
// rotation, e_q = exp(-2 pi i kq . r_n + i phi_n t) exp(-t / T2_n).
template <bool kRuns>
__device__ __forceinline__ void tc_write_b(const double *pos, const double (&kd)[kTcComps], const float *wblk,
                                           int node0, int VG, int row, int Qt, int half, uint32_t b_tile,
                                           uint32_t d_lo, uint32_t d_im) {
  F2 er[4], ei[4], ni[4];  // node pairs; ni = -ei
  const float *rate = wblk + 2 * VG * kWStride + node0;  // kRuns: 1 / T2, then phi in cycles
  const double *ph = reinterpret_cast<const double *>(wblk + 2 * (VG + 1) * kWStride) + node0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float c0, s0, c1, s1;
    tc_phase2<kRuns>(pos + 2 * i, kd, ph + 2 * i, c0, s0, c1, s1);
    if (kRuns) {
      const float2 inv = *reinterpret_cast<const float2 *>(rate + 2 * i);
      const float t = (float)kd[3], d0 = __expf(-t * inv.x), d1 = __expf(-t * inv.y);
      c0 *= d0; s0 *= d0;
      c1 *= d1; s1 *= d1;
    }
    er[i] = f2(c0, c1);
    ni[i] = f2(s0, s1);
    ei[i] = f2(-s0, -s1);
  }
  const float *wp = wblk + node0;
#pragma unroll 1
  for (int v = 0; v < VG; ++v, row += Qt, wp += 2 * kWStride) {
    const float4 *wr4 = reinterpret_cast<const float4 *>(wp), *wi4 = reinterpret_cast<const float4 *>(wp + kWStride);
    const uint32_t b = b_tile + sw64_offset(row, 16 * half);
    const int d_k2 = ((row >> 1) & 1) != 0 ? -16 : 16;
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // four nodes: one 16-byte chunk of each tile
      const float4 wr = wr4[i], wi = wi4[i];
      uint32_t h[4], l[4], hm[4], lm[4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const F2 r2 = j ? f2(wr.z, wr.w) : f2(wr.x, wr.y), i2 = j ? f2(wi.z, wi.w) : f2(wi.x, wi.y);
        const int k = 2 * i + j;
        float b0r, b1r, b0i, b1i;
        f2_get(f2_fma(er[k], r2, f2_mul(ni[k], i2)), b0r, b1r);
        f2_get(f2_fma(er[k], i2, f2_mul(ei[k], r2)), b0i, b1i);
        split_pair_im(b0r, b0i, h[2 * j], l[2 * j], hm[2 * j], lm[2 * j]);
        split_pair_im(b1r, b1i, h[2 * j + 1], l[2 * j + 1], hm[2 * j + 1], lm[2 * j + 1]);
      }
      const uint32_t at = b + (i ? d_k2 : 0);
      st_shared_v4(at, h[0], h[1], h[2], h[3]);
      st_shared_v4(at + d_lo, l[0], l[1], l[2], l[3]);
      st_shared_v4(at + d_im, hm[0], hm[1], hm[2], hm[3]);
      st_shared_v4(at + d_im + d_lo, lm[0], lm[1], lm[2], lm[3]);
    }
  }
}

// B'^T rows of a generic unit: B is only the weights of the VG columns.  The
// four A warps of a stage write it, one element a lane: column lane % 8, node
// 4 (warp % 4) + lane / 8 (a warp of its own took 700 cycles a stage for it,
// the whole of A takes 600).
__device__ __forceinline__ void tc_write_b_generic(const float *w, int VG, int quad, uint32_t b_tile, uint32_t d_lo,
                                                   uint32_t d_im) {
  const int lane = threadIdx.x & 31, v = lane & 7, node = 4 * quad + (lane >> 3);
  if (v >= VG) return;
  uint32_t h, l, hm, lm;
  split_pair_im(w[2 * v * kWStride + node], w[(2 * v + 1) * kWStride + node], h, l, hm, lm);
  // the im row is a multiple of 8 rows on, so its swizzle is the same
  const uint32_t b = b_tile + sw64_offset(v, 2 * node);
  st_shared(b, h);
  st_shared(b + d_lo, l);
  st_shared(b + d_im, hm);
  st_shared(b + d_im + d_lo, lm);
}

// ---- accumulator ---------------------------------------------------------

// Tensor memory (all 512 columns of the SM).  Wide tiles (NT > 128): the
// accumulator in columns [0, NT) collects all three products.  Narrow tiles
// (NT <= 128): the B hi and lo tiles are contiguous, so one MMA with
// N = 2 NT gives A_hi B_hi in columns [0, NT) and A_hi B_lo in [NT, 2 NT), and
// a second MMA adds A_lo B_hi into [0, NT): two MMAs per K step instead of
// three.  A narrow tile's MMAs cost about as much as wide ones to issue
// (the tensor core takes ~45 cycles per MMA at N <= 64 against 128 at
// N = 256), so their count, not their size, sets the pace.  The FP32 running
// sum follows at column sum_col.  In each part, column j < NT/2 is the real
// part of pair j and column NT/2 + j its imaginary part.
constexpr uint32_t kTcTmemCols = 512;
__host__ __device__ inline int tc_parts(int NT) { return tc_narrow(NT) ? 2 : 1; }
__host__ __device__ inline int tc_sum_col(int NT) { return ((tc_parts(NT) * NT) + 31) & ~31; }

// Folds the accumulator (complete) into the running sum: sum = part_0
// (+ part_1) for the first group, else sum + (part_0 (+ part_1)), in FP32
// round-to-nearest.  Warps 0-7: warp w handles TMEM lanes of quarter w % 4
// and every other 8 columns.
// Waits for the group (accfull, `parity`) and hands the accumulator back.  Not
// inlined: it runs once in 32 stages, and its registers would be the stage
// loops'.
__device__ __noinline__ void tc_fold(TcBars *bars, uint32_t parity, int NT, uint32_t tmem, bool first,
                                     volatile int *abort_flag) {
  const int warp = threadIdx.x >> 5;
  tc_wait(&bars->accfull, parity, abort_flag);
  __syncwarp();
  ptx::tc_fence_after();
  const int sum_col = tc_sum_col(NT);
  const bool narrow = tc_narrow(NT);
  const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 2
  for (int c0 = (warp >> 2) * 8; c0 < NT; c0 += 16) {
    uint32_t a[8], b[8], r[8];
    ptx::tmem_ld8(base + (uint32_t)c0, a);
    if (narrow) ptx::tmem_ld8(base + (uint32_t)(NT + c0), b);
    if (!first) ptx::tmem_ld8(base + (uint32_t)(sum_col + c0), r);
    ptx::tmem_wait_ld();
    if (narrow) {
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
    }
    if (!first) {
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(a[i]));
    }
    ptx::tmem_st8(base + (uint32_t)(sum_col + c0), a);
  }
  ptx::tmem_wait_st();
  ptx::tc_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(&bars->accfree);
}

// Writes the unit's result: running sum (when earlier groups were folded) +
// the accumulator of the last group (its parts added in order), to the output
// samples.  Warps 0-7: warp w reads TMEM lanes of quarter w % 4 and every
// other chunk of 8 pairs.
__device__ __forceinline__ void tc_final(const TcDev &p, const TcWork &W, const TcUnit &U, uint32_t tmem,
                                         bool has_sum) {
  const int tid = threadIdx.x, warp = tid >> 5;
  ptx::tc_fence_after();
  const int quarter = warp & 3;
  const int row = quarter * 32 + (tid & 31);
  const int NH = p.NT >> 1, VG = p.VG;
  const bool row_ok = row < U.rows;
  float2 *dst = W.out + (int64_t)U.split * p.S * p.V;
  const int Qt = p.Qt, n_pairs = Qt * VG;  // pair j: column v = j / Qt, q = j % Qt
  int64_t s_row = 0, s_q = 0;
  if (row_ok) tc_out_sample(p, U, row, s_row, s_q);
  const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
  const int n_acc = tc_parts(p.NT), AW = p.NT, sum_col = tc_sum_col(p.NT);
  for (int c0 = (warp >> 2) * 8; c0 < n_pairs; c0 += 16) {
    uint32_t r[8], m[8];
    ptx::tmem_ld8(taddr + (uint32_t)c0, r);
    ptx::tmem_ld8(taddr + (uint32_t)(NH + c0), m);
    ptx::tmem_wait_ld();
    float re8[8], im8[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      re8[i] = __uint_as_float(r[i]);
      im8[i] = __uint_as_float(m[i]);
    }
    for (int k = 1; k < n_acc; ++k) {
      ptx::tmem_ld8(taddr + (uint32_t)(k * AW + c0), r);
      ptx::tmem_ld8(taddr + (uint32_t)(k * AW + NH + c0), m);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        re8[i] = re8[i] + __uint_as_float(r[i]);
        im8[i] = im8[i] + __uint_as_float(m[i]);
      }
    }
    if (has_sum) {
      ptx::tmem_ld8(taddr + (uint32_t)(sum_col + c0), r);
      ptx::tmem_ld8(taddr + (uint32_t)(sum_col + NH + c0), m);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        re8[i] = __uint_as_float(r[i]) + re8[i];
        im8[i] = __uint_as_float(m[i]) + im8[i];
      }
    }
    if (!row_ok) continue;
    int vv = c0 / Qt, q = c0 - vv * Qt;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (q < U.Q_tile && vv < VG) dst[(s_row + q * s_q) * p.V + p.v0 + vv] = make_float2(re8[i], im8[i]);
      if (++q == Qt) {
        q = 0;
        ++vv;
      }
    }
  }
  ptx::tc_fence_before();
}

// MMAs of one stage (first: the first stage of an accumulation group, which
// overwrites the accumulator): A_hi B_hi + A_hi B_lo + A_lo B_hi over the two
// K steps.  Called by the one thread that issues every MMA and commit.
template <bool kNarrow>
__device__ __forceinline__ void tc_issue(uint32_t stage_addr, uint32_t tmem, uint32_t idesc, uint32_t idesc2,
                                         uint32_t d_blo, bool first) {
  // Shared-memory matrix descriptors: K-major operands in the 64-byte swizzled
  // layout (rows of 64 bytes, 16-byte chunks XOR-permuted by address bits 7-8,
  // 8-row groups 512 bytes apart), LBO unused (1), version 1, swizzle mode 64B (4);
  // the second K step starts 32 bytes on.  The tiles of a stage differ only in
  // the start-address field, address / 16 (below 2^14 in shared memory, and
  // every tile and stage offset a multiple of 16), so the stage's field is
  // formed once and each tile's is one add; the high word is constant.
  const uint32_t f0 = (stage_addr >> 4) | (1u << 16);                             // + LBO
  constexpr uint32_t kDescHi = (512u >> 4) | (1u << 14) | (4u << 29);            // SBO, version, 64B swizzle
  const uint32_t acc0 = first ? 0u : 1u;
  constexpr uint32_t a_lo = kAStageBytes >> 4, b_hi = 2 * kAStageBytes >> 4;
  auto desc = [&](uint32_t off) { return ((uint64_t)kDescHi << 32) | (f0 + off); };
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    // K step ks: elements 16 ks .. 16 ks + 15, bytes 32 ks .. of every row
    const uint32_t acc = ks == 0 ? acc0 : 1u;
    if (kNarrow) {
      // A_hi [B_hi; B_lo] (N = 2 NT, both tiles from b_hi on), then A_lo B_hi
      ptx::mma_bf16(tmem, desc(2 * ks), desc(b_hi + 2 * ks), idesc2, acc);
      ptx::mma_bf16(tmem, desc(a_lo + 2 * ks), desc(b_hi + 2 * ks), idesc, 1u);
    } else {
      ptx::mma_bf16(tmem, desc(2 * ks), desc(b_hi + 2 * ks), idesc, acc);
      ptx::mma_bf16(tmem, desc(2 * ks), desc(b_hi + d_blo + 2 * ks), idesc, 1u);
      ptx::mma_bf16(tmem, desc(a_lo + 2 * ks), desc(b_hi + 2 * ks), idesc, 1u);
    }
  }
}

// ---- warp roles ----------------------------------------------------------

// Warp 15, one elected thread: a stage's MMAs once its operands are written;
// each stage's slot is released by a commit to its `empty` barrier, the
// accumulator handed over by a commit to accfull after a group's last stage
// and taken back at accfree.  The election (not a test of the lane number)
// tells the compiler that one thread runs, so the descriptors go straight to
// uniform registers: an MMA issues in 40 cycles, against 100 under a lane
// predicate (whatever its shape), and a commit adds none, against 80-230.
template <bool kNarrow>
__device__ __forceinline__ bool tc_mma_unit(const TcGeom &G, TcBars *bars, uint32_t stages, uint32_t tmem, int NT,
                                            int nst, int drain, TcRing &r, uint32_t &group,
                                            volatile int *abort_flag) {
  const uint32_t idesc = ptx::idesc_bf16_f32(kTcRows, NT), idesc2 = ptx::idesc_bf16_f32(kTcRows, 2 * NT);
  int in_group = 0;  // stages of the group issued
  for (int st = 0; st < nst; ++st) {
    const bool first = in_group == 0;
    if (first && !tc_wait(&bars->accfree, (group & 1) ^ 1, abort_flag)) return false;
    if (!tc_wait(&bars->full[r.slot], r.phase, abort_flag)) return false;
    ptx::tc_fence_after();
    tc_issue<kNarrow>(stages + r.slot * G.stage_bytes, tmem, idesc, idesc2, (uint32_t)NT * 64 >> 4, first);
    ptx::mma_commit(&bars->empty[r.slot]);
    if (++in_group == drain || st == nst - 1) {
      ptx::mma_commit(&bars->accfull);
      ++group;
      in_group = 0;
    }
    r.advance(1, G.ring);
  }
  return true;
}

__device__ __forceinline__ void tc_role_mma(const TcBatchDev &B, TcBars *bars, uint32_t stages, uint32_t tmem,
                                            int n_units, volatile int *abort_flag) {
  if (ptx::elect_one()) {
    TcRing r;
    r.seek(0, B.geom.ring);
    uint32_t group = 0;
    for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
      const int e = tc_entry_of(B, u);
      const TcDev &p = B.entries[e];
      const int NT = p.NT;
      const TcUnit U = tc_unit(p, tc_work(p), u - B.offsets[e]);
      const bool ok =
          tc_narrow(NT) ? tc_mma_unit<true>(B.geom, bars, stages, tmem, NT, U.n_stages, U.drain, r, group, abort_flag)
                        : tc_mma_unit<false>(B.geom, bars, stages, tmem, NT, U.n_stages, U.drain, r, group, abort_flag);
      if (!ok) break;
    }
    // all issued MMAs complete before the tensor memory is released
    ptx::mma_commit(&bars->done);
    if (!ptx::mbar_wait(&bars->done, 0, kTcWaitNs)) *abort_flag = 1;
  }
  __syncwarp();
}

// Warps 13 and 14: the node blocks in turn, ahead of their readers; a full
// block's raw data is fetched by bulk copies into the warp's staging area while
// the other warp's block is formed.
__device__ __forceinline__ void tc_role_nodes(const TcBatchDev &B, TcBars *bars, TcMisc *misc, unsigned char *smem,
                                              int n_units, volatile int *abort_flag) {
  const int d = (threadIdx.x >> 5) - kTcNodeWarp, lane = threadIdx.x & 31;
  const TcGeom &G = B.geom;
  float *w_all = reinterpret_cast<float *>(smem + G.w);
  unsigned char *staging = smem + G.raw + d * G.raw_bytes;
  const TcRawView none{};
  uint32_t block0 = 0;  // blocks of earlier units
  uint32_t rs = 0;      // blocks staged so far by this warp
  for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
    const int e = tc_entry_of(B, u);
    const TcDev &p = B.entries[e];
    const TcUnit U = tc_unit(p, tc_work(p), u - B.offsets[e]);
    const int n_blocks = (U.n_stages + kTcStagesPerBlock - 1) / kTcStagesPerBlock;
    const TcNodeArgs a = tc_node_args(p, U, lane);
    const bool tma = p.tma != 0;
    auto n_at = [&](int blk) { return U.n_begin + (int64_t)blk * kTcBlockNodes; };
    auto staged = [&](int blk) { return tma && n_at(blk + 1) <= U.n_end; };
    auto request = [&](int blk) {
      if (blk < n_blocks && staged(blk) && lane == 0) tc_request_block(a, n_at(blk), staging, &bars->rawfull[d]);
    };
    const int first = (d + block0) & 1;
    request(first);
    TcRing nr;  // the block's node buffer
    nr.seek(block0 + first, G.node_bufs);
    for (int blk = first; blk < n_blocks; blk += 2) {
      const uint32_t b = nr.slot;
      const bool now = staged(blk);
      bool ok = tc_wait(&bars->nodeempty[b], nr.phase ^ 1, abort_flag);
      if (now) {
        // a copy in flight is waited for even where the block gives up: it must not
        // land in the shared memory of another
        if (!ptx::mbar_wait(&bars->rawfull[d], rs & 1, kTcWaitNs)) *abort_flag = 1, ok = false;
        ++rs;
      }
      if (!__all_sync(0xffffffffu, ok)) return;  // (also converges the warp: the derive exchanges values between lanes)
      int rmax = tc_derive(p, a, n_at(blk), U.n_end, now, now ? tc_raw_view(staging, a.mm_ld) : none,
                           smem + G.pos + b * kTcPosBytes, w_all + b * G.wrows * 2 * kWStride, lane);
      rmax = __reduce_max_sync(0xffffffffu, rmax);
      if (lane == 0) misc->rmax[b] = rmax;
      __syncwarp();  // the block is written and the staging area read
      if (lane == 0) ptx::mbar_arrive(&bars->nodefull[b]);
      request(blk + 2);
      nr.advance(2, G.node_bufs);
    }
    block0 += n_blocks;
  }
}

// Warps 0-12: operand tiles; warps 0-7 also fold the accumulator and write
// the results.
__device__ __forceinline__ void tc_role_operands(const TcBatchDev &B, TcBars *bars, TcMisc *misc, unsigned char *smem,
                                                 uint32_t stages, uint32_t tmem, int n_units,
                                                 volatile int *abort_flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TcGeom &G = B.geom;
  const float *w_all = reinterpret_cast<const float *>(smem + G.w);
  const uint32_t ring = G.ring, stage_bytes = G.stage_bytes;
  uint32_t stage0 = 0, group0 = 0;  // stages and accumulation groups of earlier units
  TcRing nr;                        // next node buffer
  nr.seek(0, G.node_bufs);
  for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
    const int e = tc_entry_of(B, u);
    const TcDev &p = B.entries[e];
    const TcUnit U = tc_unit(p, tc_work(p), u - B.offsets[e]);
    const int NT = p.NT, VG = p.VG, Qt = p.Qt, Q_tile = U.Q_tile, nst = U.n_stages;
    const int n_blocks = (nst + kTcStagesPerBlock - 1) / kTcStagesPerBlock;
    const bool stacked = p.stacked != 0, generic = p.kind == kTcGeneric, runs = p.kind == kTcRuns;
    const int cmask = runs ? prep_run_comps(p.ctl) : 0;  // components of k that go with the run
    const float *kc[3] = {p.kx, p.ky, p.kz};
    const bool drains = warp < kTcDrainWarps;
    // turns: three groups of A warps for a generic unit (they write its B too),
    // else two, and the other warps on B: two per stage (a node half each)
    // when the tile has more than 16 columns and there are warps for it
    const int nrg = (U.rows + 31) >> 5, a_groups = generic ? 3 : 2, nA = a_groups * nrg;
    const bool is_a = warp < nA, both = Q_tile <= 16;
    const int b_per = both || kTcOperandWarps - nA < 4 ? 1 : 2;
    const int b_groups = generic ? 0 : min((kTcOperandWarps - nA) / b_per, (int)ring);
    const uint32_t d_lo = (uint32_t)NT * 64, d_im = (uint32_t)(NT >> 1) * 64;
    // the unit's node blocks, each acquired and released in order by every
    // warp (a barrier's phases could otherwise be counted twice)
    int blk = -1, rmax = 0;
    uint32_t nbuf = 0;
    auto release = [&]() {
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->nodeempty[nbuf]);
    };
    auto acquire = [&](int to) {
      while (blk < to) {
        tc_wait(&bars->nodefull[nr.slot], nr.phase, abort_flag);
        rmax = max(rmax, misc->rmax[nr.slot]);
        nbuf = nr.slot;
        nr.advance(1, G.node_bufs);
        if (++blk < to) release();
      }
    };
    // accumulation groups folded into the running sum: group g (not the last)
    // when the ring is full of the next group's stages, so that the tensor
    // core has work as soon as the accumulator is free again
    int folded = 0;
    auto fold_before = [&](int st) {
      while (folded < U.n_groups - 1 && st >= (folded + 1) * U.drain + (int)ring - 1) {
        tc_fold(bars, (group0 + folded) & 1, NT, tmem, folded == 0, abort_flag);
        ++folded;
      }
    };
    TcRing r;
    int kmax = -1;  // |k| of this thread's phases (float bits)
    if (is_a) {
      // rows 32 rg .. of every a_groups-th stage
      const int grp = warp / nrg, rg = warp - grp * nrg, row = rg * 32 + lane;
      double kd[kTcComps] = {0, 0, 0, 0};
      int a_drow = 0;
      if (row < U.rows) {
        int rr, line;
        tc_row_line(p, U, row, rr, line);
        a_drow = 2 * (VG + rr) * kWStride;
        const int s_p = (rr == 0 ? U.start : p.start[U.it.run + rr]) + (p.kind == kTcSlab ? line * p.n_kz : line);
        // component c lies in row c, or (runs) in row tc_runs_row - 1 from row 1 on
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double k = (cmask >> c) & 1 ? 0.0 : (double)kc[c][s_p];
          const int at = runs ? tc_runs_row(cmask, c) - 1 : c;
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (i == at) kd[i] = k;
        }
        kmax = tc_abs_sum(kd[0], kd[1], kd[2]);
      }
      if (cmask) kd[2] = 1.0;  // the row of turns
      const uint32_t row_off = sw64_offset(row, 0), row_off1 = sw64_offset(row, 16);
      const int d_k2 = ((row >> 1) & 1) != 0 ? -16 : 16;
      const int arrive = rg != 0 ? 1 : kTcStageArrivals - (nrg - 1) - (generic ? 0 : b_per);
      r.seek(stage0 + grp, ring);
      for (int st = grp; st < nst; st += a_groups) {
        if (drains) fold_before(st);
        acquire(st / kTcStagesPerBlock);
        tc_wait(&bars->empty[r.slot], r.phase ^ 1, abort_flag);
        const uint32_t j = st & (kTcStagesPerBlock - 1);
        const uint32_t stg = stages + r.slot * stage_bytes;
        const float *wp = w_all + nbuf * G.wrows * 2 * kWStride + j * kTcNodes;
        if (generic)
          for (int quad = rg; quad < 4; quad += nrg)
            tc_write_b_generic(wp, VG, quad, stg + 2 * kAStageBytes, d_lo, d_im);
        const double *pos = reinterpret_cast<const double *>(smem + G.pos + nbuf * kTcPosBytes) + j * kTcNodes +
                            (runs ? kTcBlockNodes : 0);
#pragma unroll 1
        for (int n = 0; n < 16; n += 8) {
          const uint32_t addr = stg + (n ? row_off1 : row_off);
          if (stacked) tc_write_a<true>(pos + n, kd, wp + a_drow + n, addr, d_k2);
          else tc_write_a<false>(pos + n, kd, nullptr, addr, d_k2);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane < arrive) ptx::mbar_arrive(&bars->full[r.slot]);
        if (st + a_groups >= nst || (st + a_groups) / kTcStagesPerBlock > blk) release();
        r.advance(a_groups, ring);
      }
    } else {
      // the B tile of every b_groups-th stage, or a node half of it: lanes hold
      // the columns q, 32 at a time, or up to 16 of them and both node halves
      const int grp = (warp - nA) / b_per, half0 = both ? lane >> 4 : (warp - nA) - grp * b_per;
      const int lq = both ? lane & 15 : lane, half_step = both ? 2 : b_per;
      // components of k that go with the run, in the order of their rows
      const int n_run = __popc(cmask);
      const float *kr[3];
      kr[0] = cmask & 1 ? p.kx : (cmask & 2 ? p.ky : p.kz);
      kr[1] = (cmask & 3) == 3 ? p.ky : p.kz;
      kr[2] = p.kz;
      r.seek(stage0 + grp, ring);
      for (int st = grp; st < nst && grp < b_groups; st += b_groups) {
        if (drains) fold_before(st);
        acquire(st / kTcStagesPerBlock);
        tc_wait(&bars->empty[r.slot], r.phase ^ 1, abort_flag);
        const uint32_t j = st & (kTcStagesPerBlock - 1);
        const uint32_t b_tile = stages + r.slot * stage_bytes + 2 * kAStageBytes;
        const double *pos = reinterpret_cast<const double *>(smem + G.pos + nbuf * kTcPosBytes) + j * kTcNodes;
        const float *wblk = w_all + nbuf * G.wrows * 2 * kWStride;
#pragma unroll 1
        for (int q0 = 0; q0 < Q_tile; q0 += 32) {
          // lanes past the tile repeat its last column and write nothing
          const int q = min(q0 + lq, Q_tile - 1);
          const bool mine = q0 + lq < Q_tile;
          double kd[kTcComps] = {0, 0, 0, 0};
          if (runs) {
            const int s_q = p.start[U.it.q0 + q];
#pragma unroll
            for (int i = 0; i < 3; ++i) kd[i] = i < n_run ? (double)kr[i][s_q] : 0.0;
            kd[3] = p.run_t[U.it.q0 + q];
          } else {
            const int s_q = U.start + U.it.q0 + q;
            kd[0] = (double)p.kx[s_q] - (double)p.kx[U.start];
            kd[1] = (double)p.ky[s_q] - (double)p.ky[U.start];
            kd[2] = (double)p.kz[s_q] - (double)p.kz[U.start];
          }
          kmax = max(kmax, tc_abs_sum(kd[0], kd[1], kd[2]));
#pragma unroll 1
          for (int half = half0; half < 2; half += half_step) {
            if (!mine) continue;
            const int n0 = j * kTcNodes + 8 * half;
            if (runs) tc_write_b<true>(pos + 8 * half, kd, wblk, n0, VG, q, Qt, half, b_tile, d_lo, d_im);
            else tc_write_b<false>(pos + 8 * half, kd, wblk, n0, VG, q, Qt, half, b_tile, d_lo, d_im);
          }
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->full[r.slot]);
        if (st + b_groups >= nst || (st + b_groups) / kTcStagesPerBlock > blk) release();
        r.advance(b_groups, ring);
      }
    }
    while (blk < n_blocks - 1) {  // blocks past this warp's last stage
      if (drains) fold_before((blk + 1) * kTcStagesPerBlock);
      acquire(blk + 1);
      release();
    }
    // the groups that no later stage of this warp led to fold: the MMAs, and
    // with them the other warps, may wait for them
    if (drains) fold_before(nst + U.drain + (int)ring);
    // every warp has written its stages of this unit, so that none starts the
    // next unit's turns more than a round of the ring ahead of the MMAs; after a
    // wait that ran out, all leave here together
    if (ptx::named_barrier_or(2, 32 * kTcOperandWarps, *abort_flag)) break;
    // every phase of the unit had |k . r| <= kmax rmax: the fixed-point
    // reduction holds below 2^28 cycles (2^27 leaves a margin)
    if (kmax >= 0 && !((double)__int_as_float(kmax) * (double)__int_as_float(rmax) < 134217728.0))
      atomicOr(p.ctl + kCtlError, kErrPhaseRange);
    if (drains) {
      if (nst > 0) {
        tc_wait(&bars->accfull, (group0 + folded) & 1, abort_flag);
        __syncwarp();
        // the unit read again, rather than kept in registers over the loops
        const TcWork Wf = tc_work(p);
        tc_final(p, Wf, tc_unit(p, Wf, u - B.offsets[e]), tmem, folded > 0);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->accfree);
      } else if (warp < 4 && warp * 32 + lane < U.rows) {
        // no nodes in this split: its share of the tile is zero
        const TcWork W = tc_work(p);
        float2 *dst = W.out + (int64_t)U.split * p.S * p.V;
        int64_t s_row, s_q;
        tc_out_sample(p, U, warp * 32 + lane, s_row, s_q);
        for (int q = 0; q < Q_tile; ++q)
          for (int v = 0; v < VG; ++v) dst[(s_row + q * s_q) * p.V + p.v0 + v] = make_float2(0.f, 0.f);
      }
    }
    stage0 += nst;
    group0 += U.n_groups;
  }
}

__global__ void __launch_bounds__(kTcThreads, 1) signal_tc_kernel(const __grid_constant__ TcBatchDev B) {
  extern __shared__ __align__(1024) unsigned char smem[];
  // work sizes come from the device-side plan, so the launch needs no host
  // synchronisation (and can be captured in a CUDA graph)
  const int n_units = B.offsets[B.n_entries];
  const int tid = threadIdx.x, warp = tid >> 5;
  TcBars *bars = reinterpret_cast<TcBars *>(smem);
  TcMisc *misc = reinterpret_cast<TcMisc *>(smem + kTcMisc);
  volatile int *abort_flag = &misc->abort_flag;
  if (tid == 0) {
    for (int s = 0; s < kTcMaxRing; ++s) {
      ptx::mbar_init(&bars->full[s], kTcStageArrivals);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    ptx::mbar_init(&bars->accfull, 1);
    ptx::mbar_init(&bars->accfree, kTcDrainWarps);
    for (int b = 0; b < kTcMaxNodeBufs; ++b) {
      ptx::mbar_init(&bars->nodefull[b], 1);
      ptx::mbar_init(&bars->nodeempty[b], kTcOperandWarps);
    }
    for (int b = 0; b < 2; ++b) ptx::mbar_init(&bars->rawfull[b], 1);
    ptx::mbar_init(&bars->done, 1);
    misc->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) ptx::tmem_alloc(&misc->tmem, kTcTmemCols);
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *(volatile uint32_t *)&misc->tmem;
  const uint32_t stages = ptx::smem_addr(smem) + kTcFront;
  if (warp == kTcMmaWarp) tc_role_mma(B, bars, stages, tmem, n_units, abort_flag);
  else if (warp >= kTcNodeWarp) tc_role_nodes(B, bars, misc, smem, n_units, abort_flag);
  else tc_role_operands(B, bars, misc, smem, stages, tmem, n_units, abort_flag);
  ptx::tc_fence_before();
  __syncthreads();
  // a wait that ran out is reported for every problem of the launch
  if (*abort_flag)
    for (int e = tid; e < B.n_entries; e += kTcThreads) atomicOr(B.entries[e].ctl + kCtlError, kErrTimeout);
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTcTmemCols);
  }
}

// ---- plan --------------------------------------------------------------

// Node-range splits: the least estimated time of the persistent blocks, in
// stages: rounds of units times a unit's stages plus its set-up and write
// (about 12 stages), and the partial sums written and read back (a stage, about
// 0.4 us, moves some 2.6 MB).  Splits of at least 128 nodes (one node block).
__host__ __device__ inline int tc_choose_splits(int64_t items, int64_t N, int64_t outputs, int max_splits) {
  if (items <= 0) return 1;
  int best = 1;
  double best_cost = 0.0;
  for (int s = 1; s <= max_splits; ++s) {
    if (s > 1 && ceil_div(N, s) < kTcBlockNodes) break;
    const double rounds = (double)ceil_div(items * s, (int64_t)kSmCount);
    const double cost = rounds * ((double)ceil_div(ceil_div(N, s), kTcNodes) + 12.0) +
                        (s > 1 ? s * (double)outputs * 16.0 / 2.6e6 : 0.0);
    if (s == 1 || cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

// Off-resonance phases phi t that their reduction holds for (cycles_cos_sin), in
// radians: up to 2^28 cycles, and where they are added to k . r of up to 2^27 (runs
// as columns) up to 2^27.  Every node goes with every run, so the largest |phi| and
// |t| tell.
constexpr float kTcTurn = 1.6866e9f, kTcTurnRuns = 8.433e8f;
__device__ inline bool tc_turns_in_range(const TcDev &p) {
  const float turn = __int_as_float(p.ctl[kCtlPhi]) * __int_as_float(p.ctl[kCtlTime]);
  return turn < (p.use_runs && prep_static(p.ctl) ? kTcTurnRuns : kTcTurn);
}

// Node splits of every problem, shared by all its entries (from the node
// count per split when tuned, else balanced over the SMs), and the running
// unit counts of the launch's entries.  One block.
constexpr int kTcPlanThreads = 1024;
__global__ void __launch_bounds__(kTcPlanThreads) tc_plan_kernel(const TcDev *__restrict__ entries, int n,
                                                                 int split_nodes, int *__restrict__ offsets,
                                                                 int *__restrict__ first) {
  for (int e = threadIdx.x; e < n; e += kTcPlanThreads) {
    const TcDev &p = entries[e];
    if (!tc_turns_in_range(p)) atomicOr(p.ctl + kCtlError, kErrPhaseRange);
    if (e != p.first) continue;
    first[p.prob] = e;
    int splits;
    if (split_nodes > 0) {
      const int64_t s = ceil_div(p.N, (int64_t)split_nodes);
      splits = (int)(s < 1 ? 1 : (s > p.max_splits ? p.max_splits : s));
    } else {
      int64_t items = 0;
      for (int k = 0; k < p.n_of; ++k) items += tc_n_items(entries[e + k]);
      splits = tc_choose_splits(items, p.N, p.S * p.V, p.max_splits);
    }
    p.ctl[kCtlSplits] = splits;
    p.ctl[kCtlChunk] = (int)(ceil_div(ceil_div(p.N, splits), kTcNodes) * kTcNodes);
  }
  __syncthreads();
  __shared__ int part[kTcPlanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  if (threadIdx.x == 0) offsets[0] = 0;
  for (int e0 = 0; e0 < n; e0 += kTcPlanThreads) {
    const int e = e0 + threadIdx.x;
    int v = e < n ? tc_n_items(entries[e]) * *(volatile int *)(entries[e].ctl + kCtlSplits) : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= d) v += o;
    }
    __syncthreads();
    if (lane == 31) part[warp] = v;
    __syncthreads();
    int before = 0, total = 0;
    for (int i = 0; i < kTcPlanThreads / 32; ++i) {
      if (i < warp) before += part[i];
      total += part[i];
    }
    if (e < n) offsets[e + 1] = base + before + v;
    base += total;
  }
}

constexpr int kTcEntriesPerWrite = 16;
struct TcEntryChunk {
  TcDev e[kTcEntriesPerWrite];
  int n;
};

// Copies entry descriptors (passed by value) to device memory, so that the
// launch sequence holds no pointer to host memory and can be captured.
__global__ void tc_write_entries_kernel(const __grid_constant__ TcEntryChunk c, TcDev *__restrict__ dst) {
  const int words = c.n * (int)(sizeof(TcDev) / 4);
  const uint32_t *src = reinterpret_cast<const uint32_t *>(c.e);
  uint32_t *d = reinterpret_cast<uint32_t *>(dst);
  for (int i = threadIdx.x; i < words; i += blockDim.x) d[i] = src[i];
}

// Sums of the node splits, in split order, for every problem (grid y).
__global__ void tc_reduce_kernel(const TcDev *__restrict__ entries, const int *__restrict__ first) {
  const TcDev &p = entries[first[blockIdx.y]];
  const int splits = p.ctl[kCtlSplits];
  if (splits <= 1) return;
  const float2 *part = p.partials;
  const int64_t count = p.S * p.V;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (int64_t)gridDim.x * blockDim.x) {
    float2 acc = part[e];
    for (int k = 1; k < splits; ++k) {
      const float2 v = part[(int64_t)k * count + e];
      acc.x += v.x;
      acc.y += v.y;
    }
    p.out[e] = acc;
  }
}

// Workspace of one problem.
struct TcPlan {
  PrepDev prep;
  float2 *partials;
  int n_groups, max_splits;
};

// Most node splits of a problem: 16 while their partial sums stay within a
// gigabyte, more for small outputs (up to 64 in 32 MB, of a node block at least),
// which have few units.
static int tc_max_splits(int64_t S, int64_t V, int64_t N) {
  const int64_t bytes_per = S * V * 8;
  if (bytes_per <= 0) return 1;
  const int64_t s = std::min<int64_t>(16, (1LL << 30) / bytes_per);
  const int64_t small = std::min(std::min<int64_t>(64, (32LL << 20) / bytes_per), ceil_div(N, (int64_t)kTcBlockNodes));
  return (int)std::max<int64_t>(1, std::max(s, small));
}

static int tc_groups(int64_t V) { return (int)ceil_div(V, (int64_t)kTcVGroup); }

static void carve_tc(Carve &c, const fm_signal_args *a, int *ctl, TcPlan &pl) {
  const int64_t S = a->n_ro * a->n_lines * a->n_kz;
  pl.n_groups = tc_groups(a->n_vencs);
  carve_prep(c, a, kTcRows, true, kTcVGroup, sizeof(float), ctl, pl.prep);
  pl.max_splits = tc_max_splits(S, a->n_vencs, a->n_nodes);
  pl.partials = c.take<float2>((size_t)pl.max_splits * S * a->n_vencs);
}

// Entries of a launch: per problem and column group one of each kind.
static int tc_n_entries(const fm_signal_args *probs, int n) {
  int e = 0;
  for (int i = 0; i < n; ++i) e += kTcKinds * tc_groups(probs[i].n_vencs);
  return e;
}

struct TcBatchPlan {
  std::vector<TcPlan> probs;
  int *ctl;       // kCtlWords per problem
  PrepDev *prep;  // descriptors of the problems that have work
  TcDev *entries;
  int *offsets, *first;
};

static void carve_batch(Carve &c, const fm_signal_args *probs, int n, TcBatchPlan &b) {
  b.probs.resize(n > 0 ? n : 1);
  b.ctl = c.take<int>((size_t)kCtlWords * (n > 0 ? n : 1));
  b.prep = c.take<PrepDev>(n > 0 ? n : 1);
  b.first = c.take<int>(n > 0 ? n : 1);
  const int ne = tc_n_entries(probs, n);
  b.entries = c.take<TcDev>(ne > 0 ? ne : 1);
  b.offsets = c.take<int>(ne + 1);
  for (int i = 0; i < n; ++i) carve_tc(c, &probs[i], b.ctl ? b.ctl + (size_t)kCtlWords * i : nullptr, b.probs[i]);
}

// Tile shape of a column group: up to 128 (q, v) pairs per tile and at most
// 64 kz values (fewer when tuned).
static int tc_qt(const fm_signal_args *a, int VG, const fm_tc_tuning *tune) {
  int cap = (128 / VG < 64) ? 128 / VG : 64;
  if (tune && tune->kz_cap > 0 && tune->kz_cap < cap) cap = tune->kz_cap;
  return (int)((a->n_kz < cap) ? a->n_kz : cap);
}

// Columns of a tile of Qt VG pairs: real and imaginary parts.
static int tc_nt(int Qt, int VG) { return (int)ceil_div(2 * Qt * VG, 16) * 16; }

// Layout of a launch for stages of `stage_bytes`, `wrows` weight rows per node
// buffer and staging areas of raw_bytes each (ring 0 when min_ring stages and
// two node buffers do not fit).
static TcGeom tc_geom(uint32_t stage_bytes, uint32_t wrows, uint32_t raw_bytes, uint32_t min_ring = kTcMinRing) {
  TcGeom g{};
  g.stage_bytes = stage_bytes;
  g.wrows = wrows;
  g.raw_bytes = (raw_bytes + 127) & ~127u;
  const uint32_t buf = kTcPosBytes + wrows * 2 * kWStride * 4;
  const uint32_t fixed = kTcFront + 2 * g.raw_bytes;
  // as many node buffers as leave room for min_ring stages, then the stages
  for (g.node_bufs = kTcMaxNodeBufs; g.node_bufs >= kTcMinNodeBufs; --g.node_bufs)
    if (fixed + g.node_bufs * buf + min_ring * stage_bytes <= kTcSmemMax) break;
  if (g.node_bufs < kTcMinNodeBufs) return g;
  g.ring = std::min<uint32_t>(kTcMaxRing, (kTcSmemMax - fixed - g.node_bufs * buf) / stage_bytes);
  g.pos = kTcFront + g.ring * stage_bytes;
  g.w = g.pos + g.node_bufs * kTcPosBytes;
  g.raw = g.w + g.node_bufs * wrows * 2 * kWStride * 4;
  g.total = g.raw + 2 * g.raw_bytes;
  return g;
}

// Runs a stacked unit may touch, for a column group: stacking needs whole
// kz slabs within one tile and no motion (the runs then share node
// positions).  Units take 128 consecutive lines of the runs laid end to end,
// so a unit touches 128 / P runs when P divides 128, else up to
// ceil(127 / P) + 1; at most kTcMaxStack, and fewer when the node buffers (VG
// weight rows and one D row per run) would not fit in shared memory.
constexpr int kTcMaxStack = 16;
static int tc_stack_runs(const fm_signal_args *a, int VG, int Qt) {
  if (a->motion && a->motion->kind != FM_MOTION_NONE) return 1;
  if (a->n_kz < 2 || a->n_lines * a->n_kz < 2 || a->n_kz > Qt) return 1;
  const int P = (int)a->n_lines;
  int R = P >= kTcRows ? 2 : (kTcRows % P == 0 ? kTcRows / P : (kTcRows - 1 + P - 1) / P + 1);
  if (R > kTcMaxStack) R = kTcMaxStack;
  // the tiles and node buffers must fit in shared memory
  while (R > 1 && tc_geom(tc_stage_bytes(tc_nt(Qt, VG)), VG + R, 0).ring == 0) --R;
  return R < 2 ? 1 : R;
}

// Lines per stacked unit (RU) for P lines per run and units touching at most
// R runs: all 128 rows when that keeps within R runs, else whole runs
// (R P lines, units then start at run boundaries) or (R - 1) P lines (a unit
// starting inside a run then still touches at most R runs).
static int tc_pack_rows(int P, int R) {
  if ((int64_t)R * P <= kTcRows) return R * P;
  if (kTcRows % P == 0) return kTcRows;
  if ((kTcRows - 1 + P - 1) / P + 1 <= R) return kTcRows;
  return (R - 1) * P;
}

static size_t tc_batch_workspace(const fm_signal_args *probs, int n) {
  Carve c(nullptr, 0);
  TcBatchPlan b;
  carve_batch(c, probs, n, b);
  return c.used;
}

size_t tc_workspace(const fm_signal_args *a) { return tc_batch_workspace(a, 1); }

// A node's mode rows are staged up to this many modes (15 KB per block).
constexpr int kTcMaxStagedModes = 10;

// Runs per tile when runs are columns: up to 128 pairs, the tiles about equal.
static int tc_runs_qt(const fm_signal_args *a, int VG) {
  const int64_t cap = 128 / VG, tiles = ceil_div(a->n_ro, cap);
  return (int)ceil_div(a->n_ro, tiles > 0 ? tiles : 1);
}

// Whether runs as columns (where k allows it) take less time than lines x kz
// tiles: units times the time of a unit's stage, which is about 600 + 6 NT
// cycles (measured 700 at NT = 16, 2,200 at NT = 256: the A tile is always
// written in full, so wide tiles pay).
static bool tc_prefers_runs(const fm_signal_args *a, int VG, int Qt, int RU, int Qt_r) {
  auto cost = [&](int64_t units, int qt) { return units * (600 + 6 * (int64_t)tc_nt(qt, VG)); };
  const int64_t slab_units = RU > 0 ? ceil_div(a->n_ro * a->n_lines, (int64_t)RU)
                                    : a->n_ro * ceil_div(a->n_lines, (int64_t)kTcRows) * ceil_div(a->n_kz, (int64_t)Qt);
  const int64_t runs_units = ceil_div(a->n_lines * a->n_kz, (int64_t)kTcRows) * ceil_div(a->n_ro, (int64_t)Qt_r);
  if (a->n_kz < 2) return true;  // otherwise generic: one column group per 128 samples
  return cost(runs_units, Qt_r) < cost(slab_units, Qt);
}

// Launch entries of one problem; returns their number.
static int tc_entries(const fm_signal_args *a, const TcPlan &pl, const fm_tc_tuning *tune, int prob, int e0,
                      TcDev *host_entries) {
  const int64_t S = a->n_ro * a->n_lines * a->n_kz;
  const int64_t N = a->n_nodes, V = a->n_vencs;
  const PrepDev &pr = pl.prep;
  const MotionDev &md = pr.md;
  int ne = 0;
  for (int g = 0; g < pl.n_groups; ++g) {
    const int64_t v0 = (int64_t)g * kTcVGroup;
    const int VG = (int)((V - v0) < kTcVGroup ? (V - v0) : kTcVGroup);
    const int Qt_f = tc_qt(a, VG, tune);
    const int R = tc_stack_runs(a, VG, Qt_f);
    const int RU = R > 1 ? tc_pack_rows((int)a->n_lines, R) : 0;
    const int Qt_r = tc_runs_qt(a, VG);
    const int use_runs = pr.stat && tc_prefers_runs(a, VG, Qt_f, RU, Qt_r);
    for (int kind = 0; kind < kTcKinds; ++kind) {
      TcDev &p = host_entries[ne++];
      p = TcDev{};
      p.N = N; p.S = S; p.V = V;
      p.v0 = (int)v0; p.VG = VG;
      p.n_lines = (int)a->n_lines; p.n_kz = (int)a->n_kz;
      p.kx = static_cast<const float *>(a->kx);
      p.ky = static_cast<const float *>(a->ky);
      p.kz = static_cast<const float *>(a->kz);
      p.r0 = static_cast<const float *>(a->r0);
      p.phi = static_cast<const float *>(a->phi);
      p.T2 = static_cast<const float *>(a->T2);
      p.MM = static_cast<const float2 *>(pr.MM) + (size_t)g * N * kTcVGroup;
      p.mm_ld = (VG + 1) & ~1;
      p.md = md;
      p.weights = (md.kind == FM_MOTION_TERMS) ? pr.weights : nullptr;
      p.table = (a->motion && a->motion->kind == FM_MOTION_TABLE) ? static_cast<const float *>(a->motion->table)
                                                                   : nullptr;
      p.run_t = pr.run_t;
      p.start = pr.start;
      p.frun = pr.frun;
      p.tiles = pr.tiles;
      p.ctl = pr.ctl;
      p.RU = RU;
      p.prob = prob; p.first = e0; p.n_of = kTcKinds * pl.n_groups;
      p.max_splits = pl.max_splits;
      p.partials = pl.partials;
      p.out = static_cast<float2 *>(a->out);
      p.kind = kind;
      p.Qt = kind == kTcSlab ? Qt_f : (kind == kTcRuns && use_runs ? Qt_r : 1);
      // a stacked unit's node buffers add one D row per run
      const int Rk = kind == kTcSlab ? R : 1;
      p.stacked = Rk > 1 ? 1 : 0;
      p.wrows = VG + (kind == kTcRuns && use_runs ? 2 : (Rk > 1 ? Rk : 0));
      p.NT = tc_nt(p.Qt, VG);
      p.use_runs = use_runs;
      p.drain = kind == kTcRuns && !tc_narrow(p.NT) ? kTcDrainRuns : kTcDrain;
      // node blocks by bulk copies when the inputs are 16-byte aligned; the
      // mode rows of a single POD term with them (tc_batch drops either when
      // the staging areas do not fit)
      p.tma = ((uintptr_t)p.r0 % 16 == 0) && ((uintptr_t)p.T2 % 16 == 0) && ((uintptr_t)p.phi % 16 == 0) &&
              ((uintptr_t)p.MM % 16 == 0);
      if (p.tma && md.kind == FM_MOTION_TERMS && md.n_terms == 1 && md.terms[0].kind != FM_TERM_RESPIRATORY &&
          (uintptr_t)md.terms[0].modes % 16 == 0 && md.terms[0].n_modes <= kTcMaxStagedModes)
        p.mstage = 3 * md.terms[0].n_modes;
    }
  }
  return ne;
}

// Signal for n problems: per-problem preparation, then one persistent
// tensor-core launch over all of their work units, then the split sums.
static int tc_batch(fm_ctx *ctx, const fm_signal_args *probs, int n, const fm_tc_tuning *tune, void *ws,
                    size_t ws_bytes, const char *who) {
  cudaStream_t st = ctx->stream;
  Carve cv(ws, ws_bytes);
  TcBatchPlan b;
  carve_batch(cv, probs, n, b);
  FM_TRY(carve_ok(cv, who));
  std::vector<TcDev> host(tc_n_entries(probs, n) + 1);
  std::vector<fm_signal_args> work;
  std::vector<PrepDev> prep;
  int ne = 0;
  int64_t widest = 0;  // outputs of the largest problem
  for (int i = 0; i < n; ++i) {
    const fm_signal_args *a = &probs[i];
    const int64_t S = a->n_ro * a->n_lines * a->n_kz, count = S * a->n_vencs;
    if (count == 0) continue;
    if (a->n_nodes == 0) {
      FM_CUDA(cudaMemsetAsync(a->out, 0, (size_t)count * sizeof(float2), st));
      continue;
    }
    FM_REQUIRE(a->n_lines * a->n_kz < (1LL << 30), FM_ERR_SHAPE, "%s: slab too large", who);
    fill_prep(a, b.probs[i].prep);
    ne += tc_entries(a, b.probs[i], tune, (int)prep.size(), ne, host.data() + ne);
    work.push_back(*a);
    prep.push_back(b.probs[i].prep);
    if (count > widest) widest = count;
  }
  if (ne == 0) return FM_OK;
  FM_TRY(launch_prep<float>(work.data(), prep.data(), (int)prep.size(), b.prep, st));
  // one layout for all entries; staging areas (first without the mode rows,
  // then altogether) give way to the operand ring
  uint32_t stage = 0, wrows = 0, raw = 0, raw_modes = 0;
  for (int e = 0; e < ne; ++e) {
    stage = std::max(stage, tc_stage_bytes(host[e].NT));
    wrows = std::max(wrows, (uint32_t)host[e].wrows);
    if (!host[e].tma) continue;
    raw = std::max(raw, tc_raw_bytes(host[e].mm_ld));
    raw_modes = std::max(raw_modes, tc_raw_bytes(host[e].mm_ld) + tc_mode_bytes(host[e].mstage));
  }
  // in order of what costs least to give up: the mode rows' staging, the third
  // stage of slack in the ring, all staging
  TcGeom geom = tc_geom(stage, wrows, raw_modes, 4);
  if (geom.ring == 0) {
    geom = tc_geom(stage, wrows, raw, 4);
    if (geom.ring == 0) geom = tc_geom(stage, wrows, raw_modes);
    if (geom.ring == 0) geom = tc_geom(stage, wrows, raw);
    if (geom.ring == 0) geom = tc_geom(stage, wrows, 0);
  }
  for (int e = 0; e < ne; ++e) {
    if (tc_raw_bytes(host[e].mm_ld) + tc_mode_bytes(host[e].mstage) > geom.raw_bytes) host[e].mstage = 0;
    if (tc_raw_bytes(host[e].mm_ld) > geom.raw_bytes) host[e].tma = 0;
  }
  FM_REQUIRE(geom.ring != 0, FM_ERR_UNSUPPORTED, "%s: stages of %u bytes do not fit in shared memory", who, stage);
  for (int e0 = 0; e0 < ne; e0 += kTcEntriesPerWrite) {
    TcEntryChunk c;
    c.n = (ne - e0) < kTcEntriesPerWrite ? (ne - e0) : kTcEntriesPerWrite;
    for (int k = 0; k < c.n; ++k) c.e[k] = host[e0 + k];
    tc_write_entries_kernel<<<1, 256, 0, st>>>(c, b.entries + e0);
    count_launch();
    FM_TRY(check_launch("tc_write_entries_kernel"));
  }
  tc_plan_kernel<<<1, kTcPlanThreads, 0, st>>>(b.entries, ne, tune ? tune->split_nodes : 0, b.offsets, b.first);
  count_launch();
  FM_TRY(check_launch("tc_plan_kernel"));
  TcBatchDev B;
  B.entries = b.entries;
  B.offsets = b.offsets;
  B.n_entries = ne;
  B.geom = geom;
  {
    ScopedTimer timer(ctx, "signal_tc");
    FM_CUDA(cudaFuncSetAttribute(signal_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)geom.total));
    signal_tc_kernel<<<kSmCount, kTcThreads, geom.total, st>>>(B);
    count_launch();
    FM_TRY(check_launch("signal_tc_kernel"));
  }
  const int64_t rb = ceil_div(widest, 256);
  for (size_t i0 = 0; i0 < prep.size(); i0 += 65535) {
    const unsigned y = (unsigned)(prep.size() - i0 < 65535 ? prep.size() - i0 : 65535);
    tc_reduce_kernel<<<dim3((unsigned)(rb < 4 * kSmCount ? rb : 4 * kSmCount), y), 256, 0, st>>>(b.entries,
                                                                                                 b.first + i0);
    count_launch();
    FM_TRY(check_launch("tc_reduce_kernel"));
  }
  return FM_OK;
}

int signal_tc(fm_ctx *ctx, const fm_signal_args *a, void *ws, size_t ws_bytes) {
  return tc_batch(ctx, a, 1, nullptr, ws, ws_bytes, "fm_signal(BF16X3)");
}

static int tc_batch_errors(fm_ctx *ctx, const fm_signal_args *probs, int n, void *ws, size_t ws_bytes,
                           const char *who) {
  Carve cv(ws, ws_bytes);
  TcBatchPlan b;
  carve_batch(cv, probs, n, b);
  FM_TRY(carve_ok(cv, who));
  // the problems that had work, in stretches (the others' words were never set)
  int rc = FM_OK;
  bool waited = false;
  for (int i = 0; i < n;) {
    auto idle = [&](int k) {
      return probs[k].n_ro * probs[k].n_lines * probs[k].n_kz == 0 || probs[k].n_vencs == 0 || probs[k].n_nodes == 0;
    };
    if (idle(i)) {
      ++i;
      continue;
    }
    int j = i;
    while (j < n && !idle(j)) ++j;
    const int r = report_errors(b.probs[i].prep.ctl, j - i, ctx->stream, who);
    waited = true;
    if (r != FM_OK && rc == FM_OK) rc = r;
    i = j;
  }
  if (!waited) FM_CUDA(cudaStreamSynchronize(ctx->stream));
  return rc;
}

int signal_tc_errors(fm_ctx *ctx, const fm_signal_args *a, void *ws, size_t ws_bytes) {
  return tc_batch_errors(ctx, a, 1, ws, ws_bytes, "fm_signal(BF16X3)");
}

int signal_tc_batch(fm_ctx *ctx, const fm_signal_args *probs, int n, const fm_tc_tuning *tune, void *ws,
                    size_t ws_bytes) {
  return tc_batch(ctx, probs, n, tune, ws, ws_bytes, "fm_signal_batch");
}

int signal_tc_batch_errors(fm_ctx *ctx, const fm_signal_args *probs, int n, void *ws, size_t ws_bytes) {
  return tc_batch_errors(ctx, probs, n, ws, ws_bytes, "fm_signal_batch");
}

size_t tc_batch_workspace_size(const fm_signal_args *probs, int n) { return tc_batch_workspace(probs, n); }

}  // namespace fm
