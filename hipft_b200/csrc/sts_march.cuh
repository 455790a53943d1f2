// Four RKG2/RKL2 stages per pass over the field.
//
// Stages k..k+3 of diffusion_step_sts_cd (src/hipft.f90:5222-5237) with the
// 5-point operator of diffusion_operator_cd (src/hipft.f90:7927-7984), in two
// kernels that run side by side:
//
//  * k_sts_march, the rows whose four stages never reach a pole row: one warp
//    marches along phi over a strip of theta rows and keeps the stages'
//    windows in registers;
//  * k_sts_poles, the four rows next to each pole: their stages need the pole
//    ring sums of every stage over all phi columns (src/hipft.f90:7969-7979),
//    so one thread-block cluster per realization and pole holds the strip in
//    shared memory and reduces the sums through distributed shared memory.
//
// A super-step of s stages takes ceil(s / 4) passes.  Its stages are
// numbered from the back: the last pass ends with stage s, and the slots of
// the first pass before stage 1 leave Y = u0 (s is odd, so one or three of
// them).  Stage 1 (src/hipft.f90:5211-5218) is the combine with only u0 and
// dty0.  The first pass therefore reads u0 and dty0 alone.
//
// Every cell value is computed by the expressions of the single-stage
// operator in their order, whatever strip, chunk or pass it falls in, so the
// fields do not depend on how the stages are grouped.
#pragma once

#include <cooperative_groups.h>

#include "kernels.cuh"

namespace hipft {

// Coefficient tables, in load_diffusion_matrix's operation order
// (src/hipft.f90:6880-6920) for a per-realization constant D:
//   rows    [nr][3][LR]: entry jj of the three arrays holds theta row j = jj-1:
//           st_i(j), Dh dth_i(j) dt_i(j) st_i(j) sth(j), Dh dth_i(j+1) dt_i(j) st_i(j) sth(j+1)
//           for 2 <= j <= ntm-1, zeros elsewhere;
//   columns [nr][LC][2]: entry kk >= -kColPad holds phi column kk mapped onto the interior
//           column kw in 2..npm-1 it duplicates: {Dh dph_i(kw) dp_i(kw), Dh dph_i(kw+1) dp_i(kw)}.
constexpr int kColPad = 8;  // entries before column 0 and after column npm
struct PairTables {
  const double *row, *col;  // k_pair_tables output; col points at entry 0 of the first realization
  int LR, LC;               // entries per realization
};

__global__ void k_pair_tables(Mesh m, const double *__restrict__ dfac, int LR, int LC, double *rowtab,
                              double *coltab) {
  const int64_t nrow = (int64_t)m.nr * LR, ncol = (int64_t)m.nr * LC;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nrow + ncol;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < nrow) {
      const int i = (int)(e / LR) + 1, j = (int)(e % LR) - 1;
      const double Dr = dfac[i];
      const double Dh = kHalf * (Dr + Dr);
      double st = 0.0, c2 = 0.0, c4 = 0.0;
      if (j >= 2 && j <= m.ntm - 1) {
        st = m.st_i[j];
        c2 = Dh * m.dth_i[j] * m.dt_i[j] * st * m.sth[j];
        c4 = Dh * m.dth_i[j + 1] * m.dt_i[j] * st * m.sth[j + 1];
      }
      double *o = rowtab + (int64_t)(i - 1) * 3 * LR + (e % LR);
      o[0] = st;
      o[LR] = c2;
      o[2 * LR] = c4;
    } else {
      const int64_t f = e - nrow;
      const int i = (int)(f / LC) + 1, kk = (int)(f % LC) - kColPad;
      const int n2 = m.npm - 2;
      const int kw = ((kk - 2) % n2 + n2) % n2 + 2;
      const double Dr = dfac[i];
      const double Dh = kHalf * (Dr + Dr);
      coltab[2 * f] = Dh * m.dph_i[kw] * m.dp_i[kw];
      coltab[2 * f + 1] = Dh * m.dph_i[kw + 1] * m.dp_i[kw];
    }
  }
}

// Exercises the error path of the bounded waits: waits for phase 0 of an
// mbarrier that expects one arrival nobody makes, gives up after `limit`
// polls, sets the error flag and returns.
__global__ void k_wait_selftest(uint32_t limit, int *err) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (!mbar_wait_bounded(&bar, 0, limit) && threadIdx.x == 0) atomicExch(err, 1);
}

// ------------------------------------------------------------ one pass
constexpr int kMS = 4;                      // stages per pass
constexpr int kMOwn = 64 - 2 * kMS;         // theta rows a strip owns of the 64 it holds
constexpr int kMWarps = 4;                  // warps per block of k_sts_march
constexpr int kMBlocks = 3;                 // its blocks per SM (at most 168 registers)
constexpr int kMGroup = 4;                  // columns per turn of its loop
constexpr int kMSlots = 2 * kMGroup;        // columns of its shared-memory ring
constexpr int kMRing = kMSlots * 4 * 64;    // doubles per warp: Y_{k-1}, Y_{k-2}, u0, dty0
constexpr int kMCoef = 5 * kMS;             // the pass's stage coefficients
constexpr int kMColsMax = 96;               // most columns per warp
constexpr int kMTab = 2 * (kMColsMax + 2 * kMS + kMGroup);  // doubles of the column table per warp
constexpr size_t kMSmem = ((size_t)kMWarps * (kMRing + kMTab) + kMCoef) * sizeof(double);
static_assert(kMTab % 2 == 0, "16-byte aligned");
constexpr int kMBrief = 20;                 // longest chunk beside which a narrow strip's place counts (march_cols)
constexpr int kMMinRows = 2 * kMS;          // smallest ntm of the strip kernels (k_sts_whole below it)

struct MarchArgs {
  const double *x1, *x2;  // Y_{k-1}, Y_{k-2} (not read in a super-step's first pass)
  const double *u, *d;    // u0, dty0
  double *o[kMS];         // Y_k .. Y_{k+3}; null: not kept
  int first;              // this is the first pass of the super-step
  int nreal;              // realizations of the launch
  StageCoef c[kMS];       // the stages' coefficients, one set for all realizations ...
  // ... or per realization (then the launch advances the realizations in
  // rlist): rc[(i-1) * kMS + stage]
  const int *rlist;
  const StageCoef *rc;
  // steps run as a CUDA graph (with rlist and rc): the pass is *dctr + doff,
  // read on the device; dnact[pass] realizations of rlist take part and rc
  // holds dstride coefficients per pass
  const int *dctr;
  int doff;
  const int *dnact;
  int dstride;
  const int *dcols;       // ... and dcols[pass] the columns per warp
  int strips, cols;       // theta strips, columns per warp (march_cols)
  const double *dfac;     // [nr+1]
  double bcn, bcs;        // pole factors
  int *err;               // set to 1 when a bounded wait gives up
};

// Stage slot q (0-based, over the whole super-step) of an s-stage super-step
// of length dtl: stage k = q + 1 - pad, pad = the slots of the first pass
// before stage 1.
__host__ __device__ inline int64_t sts_passes(int64_t s) { return (s + kMS - 1) / kMS; }
__host__ __device__ inline StageCoef sts_slot(int method, int64_t s, int64_t q, double dtl) {
  const int64_t k = q + 1 - (kMS * sts_passes(s) - s);
  if (k < 1 || k > s) return StageCoef{0.0, 0.0, 1.0, 0.0, 0.0};
  if (k == 1) {
    double uj, vj, ubj, gj;
    sts_stage(method, s, 1, uj, vj, ubj, gj);
    return StageCoef{0.0, 0.0, 1.0, 0.0, ubj};
  }
  return sts_combine(method, s, k, dtl);
}

// Blocks and threads per block of a pole strip's cluster (k_sts_poles).
constexpr int kPMinThreads = 160, kPMidThreads = 288, kPMaxThreads = 544;
__host__ __device__ inline int poles_ranks(int n2) {
  const int per = n2 <= 8 * 152 ? 120 : 280;
  const int c = (n2 + per - 1) / per;
  return c > 8 ? 8 : c;
}
__host__ __device__ inline int poles_threads(int n2) {
  const int nc = poles_ranks(n2);
  return ((n2 + nc - 1) / nc + 2 * kMS + 31) / 32 * 32;
}
inline int poles_most_threads(int n2) {  // of the k_sts_poles that the grid takes
  const int t = poles_threads(n2);
  return t > kPMidThreads ? kPMaxThreads : t <= kPMinThreads ? kPMinThreads : kPMidThreads;
}
__host__ __device__ inline bool poles_brief(int n2) { return poles_threads(n2) <= kPMinThreads; }

// Phi columns per warp, a multiple of kMGroup: the fewest full waves of
// resident warps that keep the chunk at kMColsMax columns or less (a chunk
// loads 2 kMS columns more than it owns, so longer chunks waste less; whole
// waves leave no nearly empty one).  Blocks of k_sts_poles take the place of
// blocks; a single wave leaves those places out, which would otherwise start a
// second one.  Not where the strips' blocks are narrow (kPMinThreads) and the
// chunks would be longer than kMBrief columns: such strips end well before the
// march, and shorter chunks on all places save more than the blocks that wait for
// a strip's place lose (a super-step, places left out and not: 512x1024 x 8 2841
// and 2445 us, 359x722 x 9 939 and 840, 256x512 x 16 510 and 459; but 512x1024 x 3,
// 20 columns or 16, 1053 and 1086, and 640x1280 x 4, strips of 288 threads, 3021
// and 3609).
// A realization's chunks are dealt to its blocks' warps strip by strip: whole
// blocks per strip left up to a third of the warps without one (359x722 2.58 ->
// 2.20 us per stage, 256x512 2.30 -> 2.05).
// blocks of nw warps for the chunks of `cols` columns of one realization's strips
__host__ __device__ inline int64_t march_units(int n2, int strips, int cols, int nw) {
  const int64_t nch = (n2 + cols - 1) / cols;
  return (strips * nch + nw - 1) / nw;
}
__host__ __device__ inline int march_cols_beside(int n2, int strips, int nreal, int slots, int poles) {
  const int64_t n = nreal > 0 ? nreal : 1;
  for (int64_t w = 1;; ++w) {
    int64_t free = w * slots;
    const int64_t taken = (int64_t)poles * nreal * kMWarps;
    if (w == 1 && taken <= slots / 2) free -= taken;
    const int64_t nch = free / kMWarps / n * kMWarps / strips;  // whole blocks per realization
    if (nch < 1) continue;
    const int64_t c = ((n2 + nch - 1) / nch + kMGroup - 1) / kMGroup * kMGroup;
    if (c <= kMColsMax) return (int)c;
  }
}
__host__ __device__ inline int march_cols(int n2, int strips, int nreal, int slots, int poles) {
  const int c = march_cols_beside(n2, strips, nreal, slots, poles);
  return poles_brief(n2) && c > kMBrief ? march_cols_beside(n2, strips, nreal, slots, 0) : c;
}

// The launch's realizations and coefficients.
__device__ __forceinline__ void march_launch(const MarchArgs &a, int &nreal, bool &first, const StageCoef *&rc,
                                             int &cols) {
  nreal = a.nreal;
  first = a.first != 0;
  rc = a.rc;
  cols = a.cols;
  if (a.dctr) {
    const int p = *a.dctr + a.doff;
    nreal = a.dnact[p];
    first = p == 0;
    rc = a.rc + (int64_t)p * a.dstride;
    cols = a.dcols[p];
  }
}


__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// the shared address of this block's `a` in block `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// stores v at a shared address of the cluster and counts its 8 bytes on the
// barrier there
__device__ __forceinline__ void st_async(uint32_t dst, double v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// the same where p, of one pair of rows of four fields, kF bytes apart
template <uint32_t kF>
__device__ __forceinline__ void cp_async16x4(bool p, uint32_t dst, const void *a, const void *b, const void *c,
                                             const void *d) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n"
      " @p cp.async.cg.shared.global [%1], [%2], 16;\n @p cp.async.cg.shared.global [%1 + %6], [%3], 16;\n"
      " @p cp.async.cg.shared.global [%1 + %7], [%4], 16;\n @p cp.async.cg.shared.global [%1 + %8], [%5], 16;\n}" ::"r"(
          (uint32_t)p),
      "r"(dst), "l"(a), "l"(b), "l"(c), "l"(d), "n"(kF), "n"(2 * kF), "n"(3 * kF)
      : "memory");
}
// stores y where p, without a branch
__device__ __forceinline__ void st_if(bool p, void *g, double2 y) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p st.global.v2.f64 [%1], {%2, %3};\n}" ::"r"((uint32_t)p),
               "l"(g), "d"(y.x), "d"(y.y)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ double2 lds2(uint32_t a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}

template <int N>
struct IntC {
  static constexpr int value = N;
};

// phi-neighbour coefficients and the diagonal of a row pair in one column
struct PhiCoef {
  double2 c1, c3, c5;
};
__device__ __forceinline__ PhiCoef phi_coef(double2 st, double2 c2, double2 c4, double2 P) {
  PhiCoef r;
  r.c1 = make_double2(P.x * st.x * st.x, P.x * st.y * st.y);
  r.c5 = make_double2(P.y * st.x * st.x, P.y * st.y * st.y);
  r.c3 = make_double2(-(r.c1.x + c2.x + c4.x + r.c5.x), -(r.c1.y + c2.y + c4.y + r.c5.y));
  return r;
}

// One stage of a row pair (a, a+1) in one column: xl, xc, xr the stage input
// in columns c-1, c, c+1; up, dn the rows a-1 and a+2 of column c; o2 the
// combine's second input.
__device__ __forceinline__ double2 pair_stage(double2 xl, double2 xc, double2 xr, double up, double dn,
                                              const PhiCoef &c, double2 c2, double2 c4, double2 o2, double2 u,
                                              double2 d, const StageCoef &sc) {
  const double ax = c.c1.x * xl.x + c2.x * up + c.c3.x * xc.x + c4.x * xc.y + c.c5.x * xr.x;
  const double ay = c.c1.y * xl.y + c2.y * xc.x + c.c3.y * xc.y + c4.y * dn + c.c5.y * xr.y;
  return make_double2(sc.a * xc.x + sc.b * o2.x + sc.c * u.x + sc.d * ax + sc.e * d.x,
                      sc.a * xc.y + sc.b * o2.y + sc.c * u.y + sc.d * ay + sc.e * d.y);
}

// Four stages of the rows kMS+1 .. ntm-kMS.
//
// A warp holds 64 theta rows, two per lane, and marches along the phi columns
// of its chunk.  At the step that brings in column e of Y_{k-1}, stage k is
// computed in column e-1, stage k+1 in e-2, stage k+2 in e-3 and stage k+3 in
// e-4: each stage's input is the window of three columns that the stage before
// it left in registers, the second input is one of those as well, and the
// rows above and below come from the neighbouring lanes by shuffles.  The
// outermost rows of the strip lose one row per stage, so a strip owns the 56
// rows in its middle; strips start 56 rows apart at row 1, which makes the
// rows lost at the poles exactly those that k_sts_poles computes.  The
// column's phi coefficients are formed once and move on with the stages.
// Y_{k-1}, Y_{k-2}, u0 and dty0 arrive three columns ahead through a ring in
// shared memory, by asynchronous copies in which every lane fetches its own
// two rows: no barriers, and warps are independent.  The loop takes kMGroup
// columns per turn, so that windows, coefficients and ring slots are renamed
// and not moved.  The four warps of a block march the same columns of
// neighbouring strips where they can.  Seam columns are not written (nothing reads them in a stage).
//
// Bound: the FP64 pipe.  A pair of rows costs 4 x 36 + 14 instructions per
// column (no contraction: every product is rounded as in the reference), and
// 64/56 of that for the strip's halo; HBM sees 4 reads and 2 writes of 8 bytes
// per cell and four stages.  Where it fills the GPU, DRAM (82 % of the copy
// rate), shared memory and the FP64 pipe (69 %) are all near their ends.
// Gcell-stages/s, two stages per pass before and now: 64 x 1024x2048 165 and 393,
// 1024x2048 150 and 336; 512x1024 198, 256x512 64 (latency).
//
// TABLE: the stages' coefficients are read from shared memory.  Those of all
// realizations come as arguments, but from a chunk of more than one turn on
// they go through shared memory too: as operands from the constant bank they
// made 64 x 1024x2048 4 % and 2048x4096 6 % slower (363 and 378 against 378 and
// 399 Gcell-stages/s); a chunk of one turn does not repay the block's barrier
// (180x360: 1 % of a step).
// KEEP: Y_k and Y_{k+1} are kept too; Off: a byte offset within a
// realization's plane.
// MERGED: a pass that the GPU holds at once, in one launch: the first 2 nreal
// clusters are the pole strips, the warps of all others march.  It is then one
// grid that waits for the one before it, where the march's end would wait for
// the strips' and the next strips for the march's: 512x1024 3.16 -> 2.67 us per
// stage, 359x722 2.80 -> 2.58.  Not on narrower grids (256x512 2.30 -> 2.43:
// the strips share their SMs with the march from the start) nor where more than
// 16 columns per warp make the march the longer part.  One launch against two, a
// super-step: 361x722 x 1 to 4 0.82 to 0.86, 512x1024 0.79 and x 2 0.98, 880x880
// 0.86, 304x1216 0.98, 344x1150 x 2 0.84.  Where the march fills little more than
// half of the places two launches would take a few percent less (440x880 and
// 640x640 1.04, 210x900 1.06; 500x760 0.97, 140x700 x 3 0.90).
constexpr int kPassThreads = 160;   // most threads per block then (kPMinThreads)
constexpr int kPassColumns = 640;   // fewest phi columns
constexpr int kPassColsMax = 16;    // most columns per warp
template <int NT, bool MERGED>
__device__ __forceinline__ void poles_body(const Mesh &m, const MarchArgs &a, const PairTables &pt);

template <bool TABLE, bool KEEP, typename Off, bool MERGED>
__global__ void __launch_bounds__(MERGED ? kPassThreads : 32 * kMWarps, MERGED ? 2 : kMBlocks)
    k_sts_march(Mesh m, MarchArgs a, PairTables pt) {
  extern __shared__ __align__(16) double msm[];
  pdl_trigger();  // the next pass's blocks may take their place on the SMs; they wait for this grid's end
  const int np = MERGED ? 2 * a.nreal * (int)cooperative_groups::this_cluster().num_blocks() : 0;
  if (MERGED && (int)blockIdx.x < np) {
    poles_body<kPassThreads, true>(m, a, pt);
    return;
  }
  const unsigned block = blockIdx.x - np;
  const int nw = MERGED ? (int)blockDim.x >> 5 : kMWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npm = m.npm, n2 = npm - 2, ntm = m.ntm;
  int nreal;
  bool first;
  const StageCoef *rc;
  int ncol;
  march_launch(a, nreal, first, rc, ncol);
  // the realization's chunks, strip by strip, over its blocks' warps
  const unsigned nblk = (unsigned)march_units(n2, a.strips, ncol, nw), real = block / nblk;
  const unsigned unit = (block % nblk) * nw + warp;
  const int strip = unit % a.strips;
  const int c0 = 2 + (int)(unit / a.strips) * ncol, c1 = min(c0 + ncol - 1, npm - 1);
  if ((int)real >= nreal) {
    pdl_wait();
    return;
  }
  const int i = a.rlist ? a.rlist[real] : (int)real;  // 0-based
  double *coef = msm + nw * (kMRing + kMTab);
  if (TABLE) {
    if (threadIdx.x < kMCoef)
      coef[threadIdx.x] = a.rc ? reinterpret_cast<const double *>(rc + (int64_t)i * kMS)[threadIdx.x]
                               : reinterpret_cast<const double *>(a.c)[threadIdx.x];
    __syncthreads();
  }
  if (c0 > npm - 1) {
    pdl_wait();
    return;
  }
  const int r = 1 + kMOwn * strip + 2 * lane;  // this lane's rows r, r+1
  const double *R = pt.row + (int64_t)i * 3 * pt.LR;  // entry jj holds row jj-1
  const int e0 = min(r + 1, pt.LR - 1), e1 = min(r + 2, pt.LR - 1);
  const double2 st = make_double2(R[e0], R[e1]);
  const double2 c2 = make_double2(R[pt.LR + e0], R[pt.LR + e1]);
  const double2 c4 = make_double2(R[2 * pt.LR + e0], R[2 * pt.LR + e1]);
  const bool own = lane >= kMS / 2 && lane < 32 - kMS / 2;
  const bool va = own && r <= ntm - kMS, vb = own && r + 1 <= ntm - kMS;

  // byte offsets within the realization's plane; rows past the end of the
  // column repeat its last pair (no owned row reads them)
  const int64_t pb = (int64_t)i * m.plane;
  const Off ldb = (Off)m.ldt * 8;
  const Off rowb = (Off)min(r - 1, m.ldt - 2) * 8;
  const char *gx1 = reinterpret_cast<const char *>((first ? a.u : a.x1) + pb);
  const char *gx2 = reinterpret_cast<const char *>((first ? a.u : a.x2) + pb);
  const char *gu = reinterpret_cast<const char *>(a.u + pb), *gd = reinterpret_cast<const char *>(a.d + pb);
  const double2 *pt_col = reinterpret_cast<const double2 *>(pt.col) + (int64_t)i * pt.LC;
  char *o0 = reinterpret_cast<char *>(a.o[0] + pb), *o1 = reinterpret_cast<char *>(a.o[1] + pb);
  char *o2 = reinterpret_cast<char *>(a.o[2] + pb), *o3 = reinterpret_cast<char *>(a.o[3] + pb);
  const bool k0keep = KEEP && a.o[0], k1keep = KEEP && a.o[1];

  constexpr uint32_t kF = 512, kSlot = 4 * kF;  // bytes of one field in a slot, of a slot
  const uint32_t sring = smem_addr(msm) + (uint32_t)warp * (kMRing * 8) + 16u * lane;
  // column to fetch next, its offset, and the columns left to fetch
  int fc = c0 - kMS, left = c1 - c0 + 1 + 2 * kMS;
  if (fc < 2) fc += n2;
  Off fo = (Off)(fc - 1) * ldb + rowb;
  auto fetch = [&](uint32_t s) {
    cp_async16x4<kF>(left > 0, s, gx1 + fo, gx2 + fo, gu + fo, gd + fo);
    cp_async_commit();
    --left;
    fo += ldb;
    if (++fc > npm - 1) {
      fc = 2;
      fo -= (Off)n2 * ldb;
    }
  };
  // the column table's entries of the chunk, with the first columns' copies
  double *tab = msm + nw * kMRing + warp * kMTab;
  for (int t = lane; t < left + kMGroup - 1; t += 32) cp_async16(smem_addr(tab) + 16u * t, pt_col + c0 - kMS + t);
  // What the pass before wrote.  A merged pass waits for that pass here.  Two
  // launches: the strips' blocks trigger this grid only behind their own wait for
  // the pass before, so it has ended; that holds while the strips' launch comes
  // directly before this one and their trigger behind their wait.
  if (MERGED) pdl_wait();
  fetch(sring);
  fetch(sring + kSlot);
  fetch(sring + 2 * kSlot);

  // an odd last row: its lane stores one value of the pair
  const bool odd = strip == a.strips - 1 && ((ntm - kMS) & 1);
  auto put = [&](bool p, char *o, Off off, double2 y) {
    st_if(p && vb, o + off, y);
    if (odd && p && va && !vb) *reinterpret_cast<double *>(o + off) = y.x;
  };
  // Step of column e = the j-th of its group (compile-time j, n = step number
  // while the windows fill): W[s] holds columns e-2, e-1 of stage s's input
  // at W[s][j & 1], W[s][1 - (j & 1)], K[q & 3] the phi coefficients of the
  // column at position q of the turn; sa, sb: this turn's and the other half
  // of the ring.
  double2 W[kMS][2] = {};
  PhiCoef K[4] = {};
  int oc = -2 * kMS;                               // column e-4, counted from c0
  Off wo = (Off)(c0 - 1 - 2 * kMS) * ldb + rowb;   // its offset
  const int nown = c1 - c0 + 1;
  uint32_t ptab = smem_addr(tab);                  // the entry of column e-1
  auto step = [&](auto jc, auto nc, uint32_t sa, uint32_t sb) {
    constexpr int j = decltype(jc)::value, n = decltype(nc)::value;  // n: 2 kMS and more: all stages
    constexpr int A = j & 1, B = 1 - A;
    auto slot = [&](int back) { return j >= back ? sa + (uint32_t)(j - back) * kSlot : sb + (uint32_t)(j - back + kMGroup) * kSlot; };
    cp_async_wait<2>();
    fetch(j + 3 < kMGroup ? sa + (j + 3) * kSlot : sb + (j + 3 - kMGroup) * kSlot);  // column e-5's slot
    const double2 x0 = lds2(slot(0));
    if (n == 0) __syncwarp();  // the table was fetched by all lanes
    if (n >= 2) K[(j + 3) & 3] = phi_coef(st, c2, c4, lds2(ptab));
    if (n >= 1) ptab += 16;
    const StageCoef *q = TABLE ? reinterpret_cast<const StageCoef *>(coef) : a.c;
    double2 y0 = {}, y1 = {}, y2 = {}, y3 = {};
    if (n >= 2) {
      const uint32_t s = slot(1);
      const double2 xc = W[0][B];
      const double up = __shfl_up_sync(0xffffffffu, xc.y, 1), dn = __shfl_down_sync(0xffffffffu, xc.x, 1);
      y0 = pair_stage(W[0][A], xc, x0, up, dn, K[(j + 3) & 3], c2, c4, lds2(s + kF), lds2(s + 2 * kF), lds2(s + 3 * kF),
                      q[0]);
    }
    if (n >= 4) {
      const uint32_t s = slot(2);
      const double2 xc = W[1][B];
      const double up = __shfl_up_sync(0xffffffffu, xc.y, 1), dn = __shfl_down_sync(0xffffffffu, xc.x, 1);
      y1 = pair_stage(W[1][A], xc, y0, up, dn, K[(j + 2) & 3], c2, c4, W[0][A], lds2(s + 2 * kF), lds2(s + 3 * kF), q[1]);
    }
    if (n >= 6) {
      const uint32_t s = slot(3);
      const double2 xc = W[2][B];
      const double up = __shfl_up_sync(0xffffffffu, xc.y, 1), dn = __shfl_down_sync(0xffffffffu, xc.x, 1);
      y2 = pair_stage(W[2][A], xc, y1, up, dn, K[(j + 1) & 3], c2, c4, W[1][A], lds2(s + 2 * kF), lds2(s + 3 * kF), q[2]);
    }
    if (n >= 8) {
      const uint32_t s = slot(4);
      const double2 xc = W[3][B];
      const double up = __shfl_up_sync(0xffffffffu, xc.y, 1), dn = __shfl_down_sync(0xffffffffu, xc.x, 1);
      y3 = pair_stage(W[3][A], xc, y2, up, dn, K[j & 3], c2, c4, W[2][A], lds2(s + 2 * kF), lds2(s + 3 * kF), q[3]);
    }
    // all stores at the end: the four stages stay in one block of instructions
    if (KEEP && n >= 5 && k0keep) put(oc + 3 < nown, o0, wo + 3 * ldb, y0);
    if (KEEP && n >= 6 && k1keep) put(oc + 2 < nown, o1, wo + 2 * ldb, y1);
    if (n >= 7) put(oc + 1 < nown, o2, wo + ldb, y2);
    if (n >= 8) put(oc < nown, o3, wo, y3);
    W[0][A] = x0;
    W[1][A] = y0;
    W[2][A] = y1;
    W[3][A] = y2;
    ++oc;
    wo += ldb;
  };
  uint32_t sa = sring, sb = sring + kMGroup * kSlot;
  step(IntC<0>{}, IntC<0>{}, sa, sb);
  step(IntC<1>{}, IntC<1>{}, sa, sb);
  step(IntC<2>{}, IntC<2>{}, sa, sb);
  step(IntC<3>{}, IntC<3>{}, sa, sb);
  step(IntC<0>{}, IntC<4>{}, sb, sa);
  step(IntC<1>{}, IntC<5>{}, sb, sa);
  step(IntC<2>{}, IntC<6>{}, sb, sa);
  step(IntC<3>{}, IntC<7>{}, sb, sa);
#pragma unroll 1
  for (int t = 0; t < nown; t += kMGroup) {
    step(IntC<0>{}, IntC<8>{}, sa, sb);
    step(IntC<1>{}, IntC<8>{}, sa, sb);
    step(IntC<2>{}, IntC<8>{}, sa, sb);
    step(IntC<3>{}, IntC<8>{}, sa, sb);
    const uint32_t x = sa;
    sa = sb;
    sb = x;
  }
  cp_async_wait<0>();
  // this grid ends after the pole strips' grid, so that the next pass, which
  // waits for this one, has both
  if (!MERGED) pdl_wait();
}

// Four stages of the rows 1..kMS and ntm-kMS+1..ntm: one cluster per
// realization and pole, whose blocks share the phi columns, each with a halo
// of kMS columns.  Strip row q = 0..7 is theta row q+1 (north) or ntm-q
// (south); the rows still right after stage s are 0 .. 6-s.  The ring sum of a
// stage's input is summed over the columns of a warp by shuffles, and over the
// warps of all blocks by another tree that every warp evaluates for itself (the
// blocks and their columns depend on npm alone, so the sums do not depend on
// the batch).  The warps send their sums to every block as stores that count on
// a barrier there (a cluster barrier with release semantics took 700 cycles
// more per stage); the rows that do not need the sum are computed meanwhile.
constexpr int kPRows = 2 * kMS;  // strip rows of Y_{k-1}

// k_sts_poles: a thread owns one column, keeps its windows in registers and
// reads the neighbour columns from shared memory, where each stage leaves its
// output for the next.  Bound by latency: what the pass before does not change
// (u0, dty0, the tables) is fetched before the wait for it, and after it come
// one round of loads and four ring sums.  The stage loop is not unrolled: the
// kernel's code is cold in every pass, and fetching it once costs less.
//
// Columns per block: few on narrow grids, where the FP64 work of a block would
// otherwise outlast its ring sums.  NB = 3 holds the block's registers to those
// of one block of k_sts_march, so that it takes the place of one where the
// march fills the GPU (160 threads keep all they need then); NB = 1 is faster by
// itself.
__host__ __device__ inline int poles_stride(int threads) { return threads + 2; }  // 2 mod 32: no bank conflicts
constexpr int kPSmemRows = kPRows + 3 * (kPRows - 1);  // Y_{k-1}, Y_{k-2}, u0, dty0
__host__ __device__ inline size_t poles_smem(int threads) {
  return (size_t)kPSmemRows * poles_stride(threads) * sizeof(double);
}

template <int NT, bool MERGED>
__device__ __forceinline__ void poles_body(const Mesh &m, const MarchArgs &a, const PairTables &pt) {
  extern __shared__ __align__(16) double psm[];
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  __shared__ double s_sum[kMS][8 * (NT / 32)];
  __shared__ double s_row[3][kPRows];
  __shared__ double s_coef[5 * kMS];
  __shared__ uint64_t s_bar[kMS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int npm = m.npm, n2 = npm - 2, ntm = m.ntm;
  const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int unit = blockIdx.x / nc;
  const bool south = (unit & 1) != 0;
  int nreal;
  bool first;
  const StageCoef *rc;
  int cols;
  march_launch(a, nreal, first, rc, cols);
  if ((unit >> 1) >= nreal) {  // the whole cluster
    pdl_wait();
    if (!MERGED) pdl_trigger();
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < kMS; ++s) {
      mbar_init(&s_bar[s], 1);
      mbar_expect_tx(&s_bar[s], (uint32_t)(nc * nw * 8));
    }
    fence_mbar_init();
  }
  __syncwarp();
  cluster_arrive();  // waited for below: the blocks' barriers are ready
  const int i = a.rlist ? a.rlist[unit >> 1] : (unit >> 1);
  const int own = (n2 + nc - 1) / nc;
  const int kb = 2 + rank * own, nown = max(0, min(own, npm - kb));  // columns kb .. kb+nown-1
  const int w = nown + 2 * kMS;                                      // with the halo
  const int S = poles_stride(blockDim.x);
  double *sX = psm, *sY = psm + kPRows * S, *sU = sY + (kPRows - 1) * S, *sD = sU + (kPRows - 1) * S;
  const int64_t ld = m.ldt, pb = (int64_t)i * m.plane;
  auto wrap = [&](int c) {  // onto the core columns
    while (c < 2) c += n2;
    while (c > npm - 1) c -= n2;
    return c;
  };
  const int c = min(tid, w - 1), cm = max(c - 1, 0), cp = min(c + 1, w - 1);
  const bool mine = tid >= kMS && tid < kMS + nown;
  const int k = wrap(kb - kMS + c);
  const double2 P = reinterpret_cast<const double2 *>(pt.col)[(int64_t)i * pt.LC + k];
  const double dpk = m.dp[k], Dr = a.dfac[i + 1];
  // eight lanes per column fetch two fields' strips into shared memory
  const int t8 = tid & 7, q8 = south ? kPRows - 1 - t8 : t8, row8 = south ? ntm - kPRows + t8 : t8;
  auto strips = [&](const double *ga, const double *gb, double *sa, double *sb, int rows_a) {
    double v[2][kPRows];
#pragma unroll
    for (int n = 0; n < kPRows; ++n) {
      const int cc = min((tid >> 3) + n * (int)(blockDim.x >> 3), w - 1);
      const int64_t g = pb + (int64_t)(wrap(kb - kMS + cc) - 1) * ld + row8;
      v[0][n] = ga[g];
      v[1][n] = gb[g];
    }
#pragma unroll
    for (int n = 0; n < kPRows; ++n) {
      const int cc = (tid >> 3) + n * (int)(blockDim.x >> 3);
      if (q8 < rows_a) sa[q8 * S + cc] = v[0][n];
      if (q8 < kPRows - 1) sb[q8 * S + cc] = v[1][n];
    }
  };
  strips(a.u, a.d, sU, sD, kPRows - 1);
  if (tid < 3 * kPRows) {
    const int f = tid / kPRows, q = tid % kPRows, j = south ? ntm - q : q + 1;
    s_row[f][q] = pt.row[((int64_t)i * 3 + f) * pt.LR + j + 1];
  }
  if (tid < 5 * kMS) {
    const StageCoef *q = rc ? rc + (int64_t)i * kMS : a.c;
    s_coef[tid] = reinterpret_cast<const double *>(q)[tid];
  }
  // Everything below reads what the pass before this one wrote; the next
  // launch on the stream, this pass's k_sts_march, reads and writes other rows
  // and may start now.
  pdl_wait();
  if (!MERGED) pdl_trigger();
  strips(first ? a.u : a.x1, first ? a.u : a.x2, sX, sY, kPRows);
  __syncthreads();
  double x[kPRows], z[kPRows - 1];
#pragma unroll
  for (int q = 0; q < kPRows; ++q) x[q] = sX[q * S + c];
#pragma unroll
  for (int q = 0; q < kPRows - 1; ++q) z[q] = sY[q * S + c];
  cluster_wait();
  double *in = sX, *out = sY;  // the neighbours' input, and where the next stage finds its own
#pragma unroll 1
  for (int s = 0; s < kMS; ++s) {
    const StageCoef sc = reinterpret_cast<const StageCoef *>(s_coef)[s];
    // the warp's share of the input's ring sum, to every block
    double v = mine ? (Dr + Dr) * (south ? x[0] - x[1] : x[1] - x[0]) * dpk : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane < nc)
      st_async(cluster_addr(smem_addr(&s_sum[s][rank * nw + warp]), lane), v, cluster_addr(smem_addr(&s_bar[s]), lane));
    double y[kPRows - 1];
#pragma unroll
    for (int q = 1; q < kPRows - 1; ++q) {  // rows past 6-s are not used any more
      const double st = s_row[0][q], c2 = s_row[1][q], c4 = s_row[2][q];
      const double c1 = P.x * st * st;
      const double c5 = P.y * st * st;
      const double c3 = -(c1 + c2 + c4 + c5);
      const double up = south ? x[q + 1] : x[q - 1], dn = south ? x[q - 1] : x[q + 1];  // theta rows j-1, j+1
      const double ax = c1 * in[q * S + cm] + c2 * up + c3 * x[q] + c4 * dn + c5 * in[q * S + cp];
      y[q] = sc.a * x[q] + sc.b * z[q] + sc.c * sU[q * S + c] + sc.d * ax + sc.e * sD[q * S + c];
    }
    if (!mbar_wait_bounded(&s_bar[s], 0, 1u << 22)) atomicExch(a.err, 1);
    double ring = 0.0;
    for (int q = lane; q < nc * nw; q += 32) ring = ring + s_sum[s][q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ring += __shfl_xor_sync(0xffffffffu, ring, o);
    const double axp = south ? -ring * a.bcs : ring * a.bcn;
    y[0] = sc.a * x[0] + sc.b * z[0] + sc.c * sU[c] + sc.d * axp + sc.e * sD[c];
    // the neighbours' input of the next stage, over the one before this
    // stage's, which every thread has read
#pragma unroll
    for (int q = 1; q < kPRows - 1; ++q) out[q * S + tid] = y[q];
    double *o = a.o[s];
    if (mine && o) {
      double *g = o + pb + (int64_t)(k - 1) * ld + (south ? ntm - 1 : 0);
#pragma unroll
      for (int q = 0; q < kMS; ++q) g[south ? -q : q] = y[q];
    }
#pragma unroll
    for (int q = 0; q < kPRows - 1; ++q) {
      z[q] = x[q];
      x[q] = y[q];
    }
    double *t = in;
    in = out;
    out = t;
    __syncthreads();
  }
  cluster_arrive_relaxed();  // no block leaves while another may still send to it
  cluster_wait();
}

template <int NT, int NB>
__global__ void __launch_bounds__(NT, NB) k_sts_poles(Mesh m, MarchArgs a, PairTables pt) {
  poles_body<NT, false>(m, a, pt);
}

__host__ __device__ inline size_t pass_smem(int threads) {
  const size_t march = ((size_t)(threads / 32) * (kMRing + kMTab) + kMCoef) * sizeof(double);
  return march > poles_smem(threads) ? march : poles_smem(threads);
}
// The same strips where a column per thread does not suffice (more than about
// 4200 phi columns: k_sts_poles_any), and all rows of a grid with fewer than
// kMMinRows (k_sts_whole): one launch per stage, a cell per thread, eight lanes
// per column.  Every block adds up the ring sums that the launch before it left
// as a partial per block; s = -1 leaves those of the pass's input, which is not
// needed after a pass (its last stage left them).  A launch runs the stages s0
// to s1-1, more than one where a cluster has all columns.  Stage outputs stay in a
// scratch area, [column][8] twice: the third and fourth stage work in place.
// Bound by launches and latency, some 4 us per stage whatever the width.  (One
// cluster per pole took 112 us per pass at 64x8192, 65 with its strip in shared
// memory, and one block for a whole low grid 345 at 7x4096; now 31 and 20.)
constexpr int kPACols = 64;                          // columns per block
constexpr int kPACluster = 8;                        // most blocks of a cluster
constexpr int kPAThreads = kPRows * kPACols;
__host__ __device__ inline int poles_any_blocks(int n2) { return (n2 + kPACols - 1) / kPACols; }
// doubles per realization: two poles' strips, twice, and two sets of partials
__host__ __device__ inline int64_t poles_any_strips(int n2) { return (int64_t)4 * kPRows * n2; }
__host__ __device__ inline int64_t poles_any_doubles(int n2) { return poles_any_strips(n2) + 4 * poles_any_blocks(n2); }

// Sum of v over the block, in a fixed order, for all its threads.
__device__ __forceinline__ double strip_sum(double v, double *sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  v = lane < kPAThreads / 32 ? sh[lane] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <bool WHOLE>
__device__ __forceinline__ void poles_any_body(const Mesh &m, const MarchArgs &a, const PairTables &pt,
                                               double *scratch, int s0, int s1) {
  constexpr int NS = WHOLE ? 2 : 1;
  __shared__ double sh[2 * NS][kPAThreads / 32];
  const int tid = threadIdx.x, npm = m.npm, n2 = npm - 2, ntm = m.ntm, nb = gridDim.x;
  const bool south = !WHOLE && blockIdx.y == 1;
  int nreal;
  bool first;
  const StageCoef *rc;
  int cols;
  march_launch(a, nreal, first, rc, cols);
  if ((int)blockIdx.z >= nreal) {
    pdl_wait();
    pdl_trigger();
    return;
  }
  const int i = a.rlist ? a.rlist[blockIdx.z] : (int)blockIdx.z;
  // this thread's cell: strip row q = 0..7 is theta row q+1, or ntm-q at the south pole
  const int q = tid & (kPRows - 1), k = 2 + (int)blockIdx.x * kPACols + (tid >> 3);
  const bool live = k <= npm - 1 && q < (WHOLE ? ntm : kPRows);
  const int row = south ? ntm - 1 - q : q, dir = south ? -1 : 1;
  const int kl = k == 2 ? npm - 1 : k - 1, kr = k == npm - 1 ? 2 : k + 1;
  const int64_t pb = (int64_t)i * m.plane + row;
  auto at = [&](int c) { return pb + (int64_t)(c - 1) * m.ldt; };
  double st = 0.0, c2 = 0.0, c4 = 0.0, u = 0.0, d = 0.0, dp = 0.0;
  double2 P = {};
  const double Dr = a.dfac[i + 1];
  if (k <= npm - 1) dp = m.dp[k];
  if (live) {
    const double *R = pt.row + (int64_t)i * 3 * pt.LR + row + 2;
    st = R[0];
    c2 = R[pt.LR];
    c4 = R[2 * pt.LR];
    P = reinterpret_cast<const double2 *>(pt.col)[(int64_t)i * pt.LC + k];
    u = a.u[at(k)];
    d = a.d[at(k)];
  }
  const int pole = south ? 1 : 0;
  double *A = scratch + (int64_t)i * poles_any_doubles(n2) + (int64_t)pole * 2 * kPRows * n2, *B = A + (int64_t)kPRows * n2;
  double *part = scratch + (int64_t)i * poles_any_doubles(n2) + poles_any_strips(n2);
  auto parts = [&](int p, int stage) { return part + (int64_t)(2 * p + (stage & 1)) * nb; };
  const double *x1 = first ? a.u : a.x1, *x2 = first ? a.u : a.x2;
  // everything below reads what the launch before this one wrote; the march,
  // which is launched after the last stage, reads and writes other rows
  pdl_wait();
  pdl_trigger();
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    if (s > s0) {
      if (nb == 1) {
        __syncthreads();
      } else {
        cluster_arrive();
        cluster_wait();
      }
    }
    const bool inner = live && q >= 1 && q <= (WHOLE ? ntm - 2 : kPRows - 2 - s);
    const bool act = inner || (live && (q == 0 || (WHOLE && q == ntm - 1)));
    double y = 0.0;
    if (s < 0) {
      if (live) y = x1[at(k)];
    } else {
      const StageCoef sc = rc ? rc[(int64_t)i * kMS + s] : a.c[s];
      const int64_t e = (int64_t)(k - 2) * kPRows + q;
      double xc = 0.0, xl = 0.0, xr = 0.0, up = 0.0, dn = 0.0, z = 0.0;
      if (act) {
        const double *in = s == 0 ? x1 + at(k) : (s == 2 ? B : A) + e;
        const int64_t cs = s == 0 ? m.ldt : kPRows;
        const int rs = s == 0 ? dir : 1;  // to the next strip row
        xc = in[0];
        z = s == 0 ? x2[at(k)] : s == 1 ? x1[at(k)] : (s == 2 ? A : B)[e];
        if (inner) {
          xl = in[(kl - k) * cs];
          xr = in[(kr - k) * cs];
          up = in[south ? rs : -rs];
          dn = in[south ? -rs : rs];
        }
      }
      double rn = 0.0, rsum = 0.0;
#pragma unroll 4
      for (int b = tid; b < nb; b += kPAThreads) {
        rn = rn + parts(pole, s)[b];
        if (WHOLE) rsum = rsum + parts(1, s)[b];
      }
      rn = strip_sum(rn, sh[0]);
      if (WHOLE) rsum = strip_sum(rsum, sh[1]);
      double ax;
      if (inner) {
        const double c1 = P.x * st * st;
        const double c5 = P.y * st * st;
        const double c3 = -(c1 + c2 + c4 + c5);
        ax = c1 * xl + c2 * up + c3 * xc + c4 * dn + c5 * xr;
      } else if (WHOLE) {
        ax = q == 0 ? rn * a.bcn : -rsum * a.bcs;
      } else {
        ax = south ? -rn * a.bcs : rn * a.bcn;
      }
      y = sc.a * xc + sc.b * z + sc.c * u + sc.d * ax + sc.e * d;
      if (act) {
        if (s < kMS - 1) (s == 1 ? B : A)[e] = y;
        double *o = a.o[s];
        if (o && (WHOLE || q < kMS)) o[at(k)] = y;
      }
    }
    // this block's share of the next stage's ring sums
    const double dn = __shfl_down_sync(0xffffffffu, y, 1), up = __shfl_up_sync(0xffffffffu, y, 1);
    const double vn = strip_sum(live && q == 0 ? (Dr + Dr) * (south ? y - dn : dn - y) * dp : 0.0, sh[NS]);
    if (tid == 0) parts(pole, s + 1)[blockIdx.x] = vn;
    if (WHOLE) {
      const double vs = strip_sum(live && q == ntm - 1 ? (Dr + Dr) * (y - up) * dp : 0.0, sh[2 * NS - 1]);
      if (tid == 0) parts(1, s + 1)[blockIdx.x] = vs;
    }
  }
}

__global__ void __launch_bounds__(kPAThreads)
    k_sts_poles_any(Mesh m, MarchArgs a, PairTables pt, double *scratch, int s0, int s1) {
  poles_any_body<false>(m, a, pt, scratch, s0, s1);
}
__global__ void __launch_bounds__(kPAThreads)
    k_sts_whole(Mesh m, MarchArgs a, PairTables pt, double *scratch, int s0, int s1) {
  poles_any_body<true>(m, a, pt, scratch, s0, s1);
}

// d = scale * af, the first stage's dty0 (src/hipft.f90:5211) from A u0: one
// scale for the launch, or per realization (rscale[i-1], realizations of
// rlist; a negative entry: the slot does nothing).  Grid (chunks, slots).
__global__ void k_scale(int64_t plane, const double *__restrict__ af, double *d, double scale,
                        const int *__restrict__ rlist, const double *__restrict__ rscale) {
  int i = blockIdx.y;
  if (rlist) {
    i = rlist[i];
    if (i < 0) return;
    scale = rscale[i];
  }
  const double2 *s2 = reinterpret_cast<const double2 *>(af + (int64_t)i * plane);
  double2 *d2 = reinterpret_cast<double2 *>(d + (int64_t)i * plane);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < plane / 2; e += (int64_t)gridDim.x * blockDim.x) {
    const double2 v = s2[e];
    d2[e] = make_double2(scale * v.x, scale * v.y);
  }
}

}  // namespace hipft
