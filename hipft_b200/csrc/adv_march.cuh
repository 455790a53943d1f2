// One explicit advection stage with the WENO3 operator (src/hipft.f90:
// 7711-7925) and the integrator's combine (src/hipft.f90:7440-7578).
#pragma once

#include <algorithm>

#include "sts_march.cuh"

namespace hipft {

// theta rows a strip owns: a warp holds 64 rows of one strip, or 32 each of two chunks of it (hb = 2)
__host__ __device__ constexpr int adv_own(int hb) { return 64 / hb - 4; }
constexpr int kAWarps = 4;    // warps per block of k_adv_march
constexpr int kABlocks = 2;   // its blocks per SM: with 168 registers (3) the four chains of a step were not kept apart
constexpr int kASlots = 4;    // columns of its shared-memory ring
constexpr int kAWt = 12;      // weights of a theta face
constexpr int kAColsMax = 64;
// doubles of a ring slot: x and f0, for 2-D flows vt, at, vp, vp of the next
// column and ap; then, per chunk of the warp, the phi face's row of Weno::ptab and
// for 2-D flows the two vt above the strip
__host__ __device__ constexpr int adv_fields(bool flow2d) { return (flow2d ? 7 : 2) * 64; }
__host__ __device__ constexpr int adv_tab(bool flow2d) { return kPhiTab + (flow2d ? 2 : 0); }
__host__ __device__ constexpr int adv_slot(bool flow2d, int hb) { return adv_fields(flow2d) + hb * adv_tab(flow2d); }
__host__ __device__ constexpr size_t adv_smem(bool flow2d, int hb) {
  return ((size_t)kAWt * 64 + (size_t)kAWarps * kASlots * adv_slot(flow2d, hb)) * sizeof(double);
}

// WENO3 face value (weno_face) with the divisions of quot_nr; the two
// normalising divisions of each side share one reciprocal.  FaceW: 1 + D_C_MC
// (j-1), D_C_MC(j-1), D_C_MC(j), D_C_CP(j-1), 1 + D_C_CP(j), D_C_CP(j),
// then D_P_T(j-1), D_MC_T(j-1), D_M_T(j), D_CP_T(j), eps(j-1), eps(j).  The
// smoothness denominators are e = eps + 4 t^2 (4 t^2 is exact, so the fused
// form rounds as the reference's); big collects their high words: while those
// are below kBigE (2^100), and eps and the linear weights lie in
// weno_consts_ok's range, every operand, reciprocal and quotient is a normal
// double and the face equals weno_face's bit for bit (but for quot_nr's exception).
constexpr unsigned kBigE = (1023u + 100u) << 20;
struct FaceW {
  double a0, mc1, mc0, cp1, a1, cp0, pt, mct, mt, cpt, e1, e0;
};
__device__ __forceinline__ unsigned hi_word(double v) { return (unsigned)__double2hiint(v); }
// One side of N faces, operation by operation over the faces: the faces are
// independent, and their chains (two reciprocals and some thirty dependent
// operations each) hide each other's latency when they are interleaved.  The
// side's candidates are p0 = a v1 - d v0, p1 = f v1 + g v2 with differences
// d (v1 - v0), g (v2 - v1), linear weights l0, l1 and eps.
template <int N>
__device__ __forceinline__ void face_side(const double (&v0)[N], const double (&v1)[N], const double (&v2)[N],
                                          const double (&a)[N], const double (&d)[N], const double (&f)[N],
                                          const double (&g)[N], const double (&l0)[N], const double (&l1)[N],
                                          const double (&eps)[N], double (&u)[N], unsigned &big) {
  double w0[N], w1[N], y0[N], y1[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const double t0 = d[n] * (v1[n] - v0[n]), t1 = g[n] * (v2[n] - v1[n]);
    const double e0 = fma(kFour, t0 * t0, eps[n]), e1 = fma(kFour, t1 * t1, eps[n]);
    big = max(big, max(hi_word(e0), hi_word(e1)));
    w0[n] = e0 * e0;
    w1[n] = e1 * e1;
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    y0[n] = recip_nr(w0[n]);
    y1[n] = recip_nr(w1[n]);
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    w0[n] = quot_nr(l0[n], w0[n], y0[n]);
    w1[n] = quot_nr(l1[n], w1[n], y1[n]);
    y1[n] = w0[n] + w1[n];
  }
#pragma unroll
  for (int n = 0; n < N; ++n) y0[n] = recip_nr(y1[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const double p0 = a[n] * v1[n] - d[n] * v0[n];
    const double p1 = f[n] * v1[n] + g[n] * v2[n];
    u[n] = quot_nr(w0[n], y1[n], y0[n]) * p0 + quot_nr(w1[n], y1[n], y0[n]) * p1;
  }
}
// the same with the IEEE division, for the faces out of range, its weights read
// from shared memory: w[q * stride], in FaceW's order from t (theta faces) or
// in Weno::ptab's (phi faces)
__device__ __noinline__ double face_ieee(double LNm2, double LNm1, double LN0, double LPm1, double LP0, double LPp1,
                                         const double *w, int stride) {
  auto W = [&](int q) { return w[q * stride]; };
  if (stride == 1)
    return weno_face(LNm2, LNm1, LN0, LPm1, LP0, LPp1, W(0), W(1), W(2), W(3), W(4), W(5), W(6), W(7), W(8), W(9));
  return weno_face(LNm2, LNm1, LN0, LPm1, LP0, LPp1, W(1), W(2), W(3), W(5), W(6), W(7), W(8), W(9), W(10), W(11));
}

inline int adv_strips(int ntm, int hb) { return (ntm - 1 + adv_own(hb) - 1) / adv_own(hb); }  // rows up to ntm-1
// Chunks per warp in batches whose pole rows take one block: two of 32 rows where
// that is three quarters of the work of one of 64, or less, which holds for up to 29
// rows and for 62 to 85.  Four stages with one and two: 12x200 x 200 295 and 160 us
// (tiles of 32 rows before the marches 232), 29x60 x 300 157 and 98 (138), 20x40 x 500
// 143 and 92 (133), 64x128 x 100 191 and 168 (172), 80x160 x 16 41 and 35; 130x260 x 20,
// five sixths of the work, 105 and 107.
inline int adv_halves(int ntm) { return 2 * adv_strips(ntm, 2) <= 3 * adv_strips(ntm, 1) ? 2 : 1; }
// Phi columns per chunk: the fewest full waves of resident warps that keep the
// chunk at kAColsMax columns or less, and kAColsMin at least.
constexpr int kAColsMin = 2;
inline int adv_cols(int n2, int strips, int nreal, int slots, int hb) {
  const int64_t per = (int64_t)strips * nreal * kAWarps;
  for (int64_t w = 1;; ++w) {
    const int64_t nch = w * slots / per * kAWarps * hb;
    if (nch < 1) continue;
    const int64_t c = (n2 + nch - 1) / nch;
    if (c <= kAColsMax) return (int)std::max<int64_t>(c, kAColsMin);
  }
}

struct AdvArgs {
  const double *x, *f0;   // stage input; f0 in combine mode 1
  double *out;
  AdvCombine cb;
  // ragged batches: realization (0-based) of grid slice y (null: y itself; a
  // negative entry: none), and its substep, which multiplies cb.C (null: 1)
  const int *rlist;
  const double *rdt;
  int strips, cols;       // theta strips, phi columns per warp
  double bcn, bcs;        // pole factors
  int poles, pgrid;       // blocks per pole row (adv_pole_blocks), and for both rows
  int share;              // columns of a block's share
};

// The pole rows 1 and ntm of a realization's stage, whose value needs the ring
// sum of the upwind fluxes next to them over all phi columns (src/hipft.f90:
// 7902-7915): NP rows of the block, from `south0` (0: row 1) on, each added up whole,
// as 256 threads (two per thread here) and a tree over them do, and this block's
// share of the columns written.  Bound by latency and, on wide grids, by the
// sectors one SM can take in.  a.poles blocks per pole, a block per kAPole columns:
// one block for both poles, a column's loads behind the store of the one before,
// held a stage of 64x8192 up for 63 us (now 38) and of 16x2048 for 19 (now 10).
// From kAPoleBoth realizations on, one block takes both rows where one per pole
// would do: their number is what counts then (four stages, a block per row and one:
// 20x40 x 100 48.8 and 44.6 us, 12x12 x 100 30.9 and 27.4, 16x1000 x 8 67.7 and 53.9,
// 64x128 x 30 61.6 and 57.5; 33x600 x 8 39.6 and 41.1); with fewer its latency does
// (180x360 20.6 and 22.7, 90x181 18.6 and 20.6).
constexpr int kAPoleBoth = 8;
constexpr int kAPole = 1024;
inline int adv_pole_blocks(int n2, int nreal) {  // per pole
  return std::min((n2 + kAPole - 1) / kAPole, std::max(1, kDPoleMax / nreal));
}
inline int adv_pole_grid(int n2, int nreal) {  // for both rows
  const int b = adv_pole_blocks(n2, nreal);
  return b > 1 || nreal < kAPoleBoth ? 2 * b : 1;
}
template <int NP>
__device__ __forceinline__ void adv_pole_rows(const Mesh &m, const Flow &fl, const AdvArgs &a, int i0, int south0,
                                              int block, double *sh) {
  const int i = i0 + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ld = m.ldt, p0 = (int64_t)i0 * m.plane;
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    double f[NP] = {};
#pragma unroll 4
    for (int k = 2 + (int)threadIdx.x + 128 * v; k <= m.npm - 1; k += 256) {
#pragma unroll
      for (int s = 0; s < NP; ++s) {
        const bool south = south0 + s != 0;
        const double *c = a.x + p0 + (int64_t)(k - 1) * ld + (south ? m.ntm - 1 : 0);
        const double xp = c[0], xn = c[south ? -1 : 1];
        const double ft = upwind_flux(vt_at(m, fl, south ? m.nt - 1 : 2, k, i), fl.upwind, south ? xp : xn, south ? xn : xp);
        f[s] = f[s] + ft * m.dp[k];
      }
    }
#pragma unroll
    for (int s = 0; s < NP; ++s) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) f[s] += __shfl_down_sync(0xffffffffu, f[s], o);
      if (lane == 0) sh[8 * s + 4 * v + warp] = f[s];
    }
  }
  __syncthreads();
  double ax[NP];
#pragma unroll
  for (int s = 0; s < NP; ++s) {
    double f = lane < 8 ? sh[8 * s + lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f += __shfl_down_sync(0xffffffffu, f, o);
    f = __shfl_sync(0xffffffffu, f, 0);
    ax[s] = south0 + s ? -f * a.bcs : f * a.bcn;
  }
  const double C = a.rdt ? a.cb.C * a.rdt[i0] : a.cb.C;
  const int k1 = min(1 + a.share * (block + 1), m.npm - 1);
  constexpr int G = 4 / NP;  // columns per turn, their loads all under way at once
  for (int k0 = 2 + a.share * block + (int)threadIdx.x; k0 <= k1; k0 += 128 * G) {
    double xv[G][NP], fv[G][NP];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (k0 + 128 * g > k1) break;
#pragma unroll
      for (int s = 0; s < NP; ++s) {
        const int64_t p = p0 + (int64_t)(k0 + 128 * g - 1) * ld + (south0 + s ? m.ntm - 1 : 0);
        xv[g][s] = a.x[p];
        fv[g][s] = a.cb.mode == 0 ? 0.0 : a.f0[p];
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int k = k0 + 128 * g;
      if (k > k1) break;
      const int64_t sm = k == 2 ? (m.npm - 2) * ld : k == m.npm - 1 ? -(m.npm - 2) * ld : 0;
#pragma unroll
      for (int s = 0; s < NP; ++s) {
        const int64_t p = p0 + (int64_t)(k - 1) * ld + (south0 + s ? m.ntm - 1 : 0);
        const double y =
            a.cb.mode == 0 ? xv[g][s] - C * ax[s] : a.cb.A * fv[g][s] + a.cb.B * xv[g][s] - C * ax[s];
        a.out[p] = y;
        if (sm) a.out[p + sm] = y;
      }
    }
  }
}

// One stage; the first blocks of a realization take the pole rows, the others the
// rows 2..ntm-1.  A warp holds 64 theta rows, two per lane, and
// marches along the phi columns of its chunk: at the step that brings in
// column e it computes the phi faces e-1 of its rows and, for the cells of
// column k = e-2, the theta faces between its rows and above them: every face
// once, four per lane and step, as independent chains.  The phi faces' inputs
// are windows of the row in registers, the theta faces' come from the
// neighbouring lanes by shuffles, and the outermost rows of the strip only
// supply those.  Inputs arrive three columns ahead through a ring in shared
// memory, by asynchronous copies of the lane's own rows (the phi faces' table
// row by lanes 0..7); the theta faces' weights sit in shared memory, shared by
// the block's warps, which march four neighbouring chunks of one strip.  The
// next stage may be launched when this one's blocks have started; it sets up its
// tables and then waits for this one.
//
// Bound: the FP64 pipe, about 95 instructions per face and 210 per cell, most
// of them the eight divisions per face (two reciprocals shared).
//
// FLOW2D: 2-D velocities; MODE: the combine; Off: a byte offset in a plane; BOTH:
// one block for both pole rows (adv_pole_grid; code for either in one kernel made
// a stage of 512x1024 0.4 us longer).
// HB: chunks per warp (adv_halves), the second one by the upper half of its lanes.
template <bool FLOW2D, int MODE, typename Off, bool BOTH, int HB>
__global__ void __launch_bounds__(32 * kAWarps, kABlocks) k_adv_march(Mesh m, Flow fl, Weno wn, AdvArgs a) {
  extern __shared__ __align__(16) double asm_[];
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ntm = m.ntm, npm = m.npm, n2 = npm - 2, nt = m.nt;
  const int i = a.rlist ? a.rlist[blockIdx.y] : (int)blockIdx.y;  // 0-based
  if (i < 0) {
    pdl_wait();
    return;
  }
  if ((int)blockIdx.x < a.pgrid) {
    pdl_wait();
    adv_pole_rows<BOTH ? 2 : 1>(m, fl, a, i, BOTH ? 0 : (int)blockIdx.x & 1, BOTH ? 0 : (int)blockIdx.x >> 1, asm_);
    return;
  }
  const int blk = (int)blockIdx.x - a.pgrid, strip = blk % a.strips;
  constexpr int LH = 32 / HB, ROWS = 64 / HB;
  const int hl = lane & (LH - 1), half = lane / LH;
  const int R0 = adv_own(HB) * strip - 1;  // rows R0 .. R0+ROWS-1, owned: R0+2 .. R0+ROWS-3
  for (int p = threadIdx.x; p < ROWS; p += 32 * kAWarps) {
    // weights of the face above row R0+p
    const int jw = min(max(R0 + p + 1, 2), nt - 1);
    const double v[kAWt] = {kOne + wn.mct[jw - 1], wn.mct[jw - 1], wn.mct[jw], wn.cpt[jw - 1], kOne + wn.cpt[jw],
                            wn.cpt[jw],            wn.pt[jw - 1],  wn.mctt[jw - 1], wn.mt[jw], wn.cptt[jw],
                            wn.epst[jw - 1],       wn.epst[jw]};
#pragma unroll
    for (int q = 0; q < kAWt; ++q) asm_[q * 64 + p] = v[q];
  }
  __syncthreads();
  const int cw = 2 + (blk / a.strips * kAWarps + warp) * HB * a.cols, n0 = min(a.cols, npm - cw);
  if (cw > npm - 1) {
    pdl_wait();
    return;
  }
  // this lane's chunk; a second one past the end has no columns: nothing is fetched or
  // stored for it, and what its lanes compute is not looked at
  const int ch = cw + half * a.cols;
  const int c0 = ch > npm - 1 ? 2 : ch, c1 = ch > npm - 1 ? -4 : min(c0 + a.cols - 1, npm - 1);
  const double C = a.rdt ? a.cb.C * a.rdt[i] : a.cb.C;
  const int r = R0 + 2 * hl;  // this lane's rows r, r+1
  const bool own = hl >= 1 && hl <= LH - 2;
  const bool va = own && r >= 2 && r <= ntm - 1, vb = own && r + 1 <= ntm - 1;
  const bool tupA = r + 1 == 2 || r + 1 == ntm, tupB = r + 2 == 2 || r + 2 == ntm;
  const bool wup = __any_sync(0xffffffffu, tupA || tupB);
  const bool edge = __any_sync(0xffffffffu, va != vb);  // a pair stored by halves
  const uint32_t swt = smem_addr(asm_) + 16u * hl;
  bool tok;  // the weights of this lane's WENO faces (3 .. nt-2) are in range
  {
    auto ok = [&](int q) {
      const int jf = R0 + q + 1;
      const double *w = asm_ + q;
      return jf < 3 || jf > nt - 2 ||
             weno_consts_ok(w[6 * 64], w[7 * 64], w[8 * 64], w[9 * 64], w[10 * 64], w[11 * 64]);
    };
    tok = ok(2 * hl) && ok(2 * hl + 1);
  }
  // divergence factors of rows r, r+1
  const int ra = min(max(r, 1), ntm), rb = min(max(r + 1, 1), ntm);
  const double sth0 = m.sth[ra], sth1 = m.sth[min(max(r + 1, 1), nt)], sth2 = m.sth[min(max(r + 2, 1), nt)];
  const double2 sti = make_double2(m.st_i[ra], m.st_i[rb]), dti = make_double2(m.dt_i[ra], m.dt_i[rb]);
  // LN(c) = half x(c) (vt(c)+at(c)) and LP(c) = half x(c) (vt(c+1)-at(c)) are
  // formed as x(c) * (half (vt(c)+at(c))) etc.: halving is exact, so the
  // products are the reference's (for |x| above 2^-1021, i.e. any map)
  double2 tn = {}, tp = {}, pn = {}, pp = {};
  double vuA = 0.0, vuB = 0.0;  // velocities of the upwind faces r+1, r+2
  if (!FLOW2D) {
    const double *vt = fl.vt1 + (int64_t)i * (nt + 1), *at = fl.at1 + (int64_t)i * (ntm + 1);
    const double *vp = fl.vp1 + (int64_t)i * (ntm + 1), *ap = fl.ap1 + (int64_t)i * (ntm + 1);
    const double va0 = vt[ra], va1 = vt[min(max(r + 1, 1), nt)], va2 = vt[min(max(r + 2, 1), nt)];
    tn = make_double2(kHalf * (va0 + at[ra]), kHalf * (va1 + at[rb]));
    tp = make_double2(kHalf * (va1 - at[ra]), kHalf * (va2 - at[rb]));
    pn = make_double2(kHalf * (vp[ra] + ap[ra]), kHalf * (vp[rb] + ap[rb]));
    pp = make_double2(kHalf * (vp[ra] - ap[ra]), kHalf * (vp[rb] - ap[rb]));
    vuA = va1;
    vuB = va2;
  }

  // ring of input columns
  constexpr uint32_t kF = 512, kSlot = adv_slot(FLOW2D, HB) * 8;
  double *rbase = asm_ + kAWt * 64 + warp * kASlots * adv_slot(FLOW2D, HB);
  double *rtab = rbase + adv_fields(FLOW2D) + half * adv_tab(FLOW2D);
  const uint32_t sring = smem_addr(rbase) + 16u * lane, stab = smem_addr(rtab);
  const int64_t pb = (int64_t)i * m.plane, vb0 = (int64_t)i * fl.vplane;
  const Off ldb = (Off)m.ldt * 8, lvb = (Off)fl.ldv * 8;
  const Off rowb = (Off)min(max(r - 1, 0), m.ldt - 2) * 8, rowv = (Off)min(max(r - 1, 0), fl.ldv - 2) * 8;
  const char *gx = reinterpret_cast<const char *>(a.x + pb), *gf = reinterpret_cast<const char *>(a.f0 + pb);
  const char *gvt = reinterpret_cast<const char *>(fl.vt + vb0), *gat = reinterpret_cast<const char *>(fl.at + vb0);
  const char *gvp = reinterpret_cast<const char *>(fl.vp + vb0), *gap = reinterpret_cast<const char *>(fl.ap + vb0);
  char *go = reinterpret_cast<char *>(a.out + pb);
  const Off upv = r + 1 <= fl.ldv - 2 ? 16 : 0;  // to the pair of rows r+2, r+3 (not read past the faces)
  int fe = c0 - 2, fs = 0;  // column to fetch next, its slot
  auto fetch = [&]() {
    if (fe <= c1 + 2) {
      const uint32_t s = sring + fs * kSlot;
      const int cp = fe < 1 ? fe + n2 : fe > npm - 1 ? fe - n2 : fe;  // the reference's periodic pad
      cp_async16(s, gx + ((Off)(cp - 1) * ldb + rowb));
      if (FLOW2D) {
        const Off o = (Off)(cp - 1) * lvb + rowv;
        cp_async16(s + 4 * kF, gvp + o);
        cp_async16(s + 5 * kF, gvp + (o + lvb));
        cp_async16(s + 6 * kF, gap + o);
      }
      if (fe >= c0 + 1 && hl < kPhiTab / 2)
        cp_async16(stab + fs * kSlot + 16u * hl, wn.ptab + (int64_t)(fe - 3) * kPhiTab + 2 * hl);
      if (fe >= c0 + 2) {
        if (MODE != 0) cp_async16(s + kF, gf + ((Off)(fe - 3) * ldb + rowb));
        if (FLOW2D) {
          const Off o = (Off)(fe - 3) * lvb + rowv;
          cp_async16(s + 2 * kF, gvt + o);
          cp_async16(s + 3 * kF, gat + o);
          if (hl == LH - 1) cp_async16(stab + fs * kSlot + kPhiTab * 8, gvt + (o + upv));
        }
      }
    }
    cp_async_commit();
    ++fe;
    fs = (fs + 1) & (kASlots - 1);
  };
  pdl_wait();
  fetch();
  fetch();
  fetch();

  // windows at the step of column e: LN at e-3, e-2, e-1; LP and x at e-2, e-1
  double2 LN0 = {}, LN1 = {}, LN2 = {}, LP0 = {}, LP1 = {}, x0 = {}, x1 = {}, Fplo = {};
  double dpk = 0.0;
  int slot = 0;
  auto step = [&](int e, auto phc) {
    constexpr int PH = decltype(phc)::value;  // 0: fill the windows, 1: and the first phi face, 2: everything
    cp_async_wait<2>();
    __syncwarp();  // the table row came by other lanes; and the slot fetched next is read out
    fetch();
    const uint32_t s = sring + slot * kSlot, st = stab + slot * kSlot;
    slot = (slot + 1) & (kASlots - 1);
    const double2 xe = lds2(s);
    double2 cN = pn, cP = pp;
    if (FLOW2D) {
      const double2 v0 = lds2(s + 4 * kF), v1 = lds2(s + 5 * kF), al = lds2(s + 6 * kF);
      cN = make_double2(kHalf * (v0.x + al.x), kHalf * (v0.y + al.y));
      cP = make_double2(kHalf * (v1.x - al.x), kHalf * (v1.y - al.y));
    }
    const double2 LN3 = make_double2(xe.x * cN.x, xe.y * cN.y), LP2 = make_double2(xe.x * cP.x, xe.y * cP.y);
    double2 Fp = {};
    double dpn = 0.0;
    if (PH >= 1) {
      unsigned big = 0;
      const double2 q0 = lds2(st), q1 = lds2(st + 16), q2 = lds2(st + 32), q3 = lds2(st + 48), q4 = lds2(st + 64),
                    q5 = lds2(st + 80), q6 = lds2(st + 96);
      const FaceW wp{q6.x, q0.x, q0.y, q1.x, q6.y, q1.y, q2.x, q2.y, q3.x, q3.y, q4.x, q4.y};
      dpn = q5.y;
      if (PH == 1) {
        double um[2], up[2];
        face_side<2>({LN0.x, LN0.y}, {LN1.x, LN1.y}, {LN2.x, LN2.y}, {wp.a0, wp.a0}, {wp.mc1, wp.mc1}, {wp.mc0, wp.mc0},
                     {wp.cp1, wp.cp1}, {wp.pt, wp.pt}, {wp.mct, wp.mct}, {wp.e1, wp.e1}, um, big);
        face_side<2>({LP2.x, LP2.y}, {LP1.x, LP1.y}, {LP0.x, LP0.y}, {wp.a1, wp.a1}, {wp.cp0, wp.cp0}, {wp.cp1, wp.cp1},
                     {wp.mc0, wp.mc0}, {wp.mt, wp.mt}, {wp.cpt, wp.cpt}, {wp.e0, wp.e0}, up, big);
        Fp = make_double2(up[0] + um[0], up[1] + um[1]);
      }
      double FA = 0.0, FB = 0.0;
      double2 fc = {}, LNt = {}, LPt = {};
      double LNm = 0.0, LNp = 0.0, LPp = 0.0, LPq = 0.0;
      if (PH == 2) {
        double2 ctn = tn, ctp = tp;
        if (FLOW2D) {
          const double2 v = lds2(s + 2 * kF), al = lds2(s + 3 * kF);
          const double vn = __shfl_down_sync(0xffffffffu, v.x, 1);
          const double v2 = hl == LH - 1 ? lds2(st + kPhiTab * 8).x : vn;
          ctn = make_double2(kHalf * (v.x + al.x), kHalf * (v.y + al.y));
          ctp = make_double2(kHalf * (v.y - al.x), kHalf * (v2 - al.y));
          vuA = v.y;
          vuB = v2;
        }
        if (MODE != 0) fc = lds2(s + kF);
        LNt = make_double2(x0.x * ctn.x, x0.y * ctn.y);
        LPt = make_double2(x0.x * ctp.x, x0.y * ctp.y);
        LNm = __shfl_up_sync(0xffffffffu, LNt.y, 1);
        LNp = __shfl_down_sync(0xffffffffu, LNt.x, 1);
        LPp = __shfl_down_sync(0xffffffffu, LPt.x, 1);
        LPq = __shfl_down_sync(0xffffffffu, LPt.y, 1);
        double2 t[kAWt];
#pragma unroll
        for (int q = 0; q < kAWt; ++q) t[q] = lds2(swt + q * 512u);
        const FaceW wA{t[0].x, t[1].x, t[2].x, t[3].x, t[4].x, t[5].x, t[6].x, t[7].x, t[8].x, t[9].x, t[10].x, t[11].x};
        const FaceW wB{t[0].y, t[1].y, t[2].y, t[3].y, t[4].y, t[5].y, t[6].y, t[7].y, t[8].y, t[9].y, t[10].y, t[11].y};
        // the phi faces e-1 and the theta faces of column e-2
        double um[4], up[4];
        face_side<4>({LN0.x, LN0.y, LNm, LNt.x}, {LN1.x, LN1.y, LNt.x, LNt.y}, {LN2.x, LN2.y, LNt.y, LNp},
                     {wp.a0, wp.a0, wA.a0, wB.a0}, {wp.mc1, wp.mc1, wA.mc1, wB.mc1}, {wp.mc0, wp.mc0, wA.mc0, wB.mc0},
                     {wp.cp1, wp.cp1, wA.cp1, wB.cp1}, {wp.pt, wp.pt, wA.pt, wB.pt}, {wp.mct, wp.mct, wA.mct, wB.mct},
                     {wp.e1, wp.e1, wA.e1, wB.e1}, um, big);
        face_side<4>({LP2.x, LP2.y, LPp, LPq}, {LP1.x, LP1.y, LPt.y, LPp}, {LP0.x, LP0.y, LPt.x, LPt.y},
                     {wp.a1, wp.a1, wA.a1, wB.a1}, {wp.cp0, wp.cp0, wA.cp0, wB.cp0}, {wp.cp1, wp.cp1, wA.cp1, wB.cp1},
                     {wp.mc0, wp.mc0, wA.mc0, wB.mc0}, {wp.mt, wp.mt, wA.mt, wB.mt}, {wp.cpt, wp.cpt, wA.cpt, wB.cpt},
                     {wp.e0, wp.e0, wA.e0, wB.e0}, up, big);
        Fp = make_double2(up[0] + um[0], up[1] + um[1]);
        FA = up[2] + um[2];
        FB = up[3] + um[3];
      }
      if (!(big < kBigE && tok && q5.x != 0.0) && (HB == 1 || e <= c1 + 2)) {
        const double *w = rtab + ((slot + kASlots - 1) & (kASlots - 1)) * adv_slot(FLOW2D, HB);
        Fp.x = face_ieee(LN0.x, LN1.x, LN2.x, LP0.x, LP1.x, LP2.x, w, 1);
        Fp.y = face_ieee(LN0.y, LN1.y, LN2.y, LP0.y, LP1.y, LP2.y, w, 1);
        if (PH == 2) {
          FA = face_ieee(LNm, LNt.x, LNt.y, LPt.x, LPt.y, LPp, asm_ + 2 * hl, 64);
          FB = face_ieee(LNt.x, LNt.y, LNp, LPt.y, LPp, LPq, asm_ + 2 * hl + 1, 64);
        }
      }
      if (PH == 2) {
        if (wup) {  // first-order upwind next to the poles
          const double xn = __shfl_down_sync(0xffffffffu, x0.x, 1);
          if (tupA) FA = upwind_flux(vuA, fl.upwind, x0.y, x0.x);
          if (tupB) FB = upwind_flux(vuB, fl.upwind, xn, x0.y);
        }
        const double Flo = __shfl_up_sync(0xffffffffu, FB, 1);
        const double aopx = (sth1 * FA - sth0 * Flo) * sti.x * dti.x + (Fp.x - Fplo.x) * sti.x * dpk;
        const double aopy = (sth2 * FB - sth1 * FA) * sti.y * dti.y + (Fp.y - Fplo.y) * sti.y * dpk;
        const double2 y = MODE == 0 ? make_double2(x0.x - C * aopx, x0.y - C * aopy)
                                    : make_double2(a.cb.A * fc.x + a.cb.B * x0.x - C * aopx,
                                                   a.cb.A * fc.y + a.cb.B * x0.y - C * aopy);
        const int k = e - 2;
        const bool sa = va && (HB == 1 || k <= c1), sb = vb && (HB == 1 || k <= c1);
        char *g = go + ((Off)(k - 1) * ldb + rowb);
        st_if(sa && sb, g, y);
        if (edge || k == 2 || k == npm - 1) {
          const int64_t sm = k == 2 ? (int64_t)n2 * m.ldt : k == npm - 1 ? -(int64_t)n2 * m.ldt : 0;
          double *d = reinterpret_cast<double *>(g);
          if (sa) d[sm] = y.x;
          if (sb) d[sm + 1] = y.y;
          if (sa && !sb) d[0] = y.x;
          if (sb && !sa) d[1] = y.y;
        }
      }
    }
    LN0 = LN1;
    LN1 = LN2;
    LN2 = LN3;
    LP0 = LP1;
    LP1 = LP2;
    x0 = x1;
    x1 = xe;
    Fplo = Fp;
    dpk = dpn;
  };
#pragma unroll 1
  for (int e = c0 - 2; e <= c0; ++e) step(e, IntC<0>{});
  step(c0 + 1, IntC<1>{});
#pragma unroll 1
  for (int e = c0 + 2; e < c0 + 2 + n0; ++e) step(e, IntC<2>{});
  cp_async_wait<0>();
}

}  // namespace hipft
