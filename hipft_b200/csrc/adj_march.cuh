// Reverse RKG2 stages, four or two per pass, by warps that march along phi
// (k_adj_march) and a cluster per pole (k_adj_poles): the forward's passes
// (sts_march.cuh) with the transposed operator.  Stages K = k, k-1, .. of the
// reverse recurrence with w0 = W_k, w1 = W_{k+1}:
//   W_{K-1} = a W_K + b W_{K+1} + c A^T W_K,
//   ub += c0 W_K,  db += g W_K,  dpart += ds <A^T W_K, Y_{K-1}>.
// The operator has the expressions of adj_diff_at_tab in their order.
//
// Bound by latency where one field does not fill the GPU (a march's warp has
// 270 instructions per column, half of them FP64, in four dependent stages; a
// strip's block has a ring sum per stage), else by memory: 12 reads and 4 writes
// of 8 bytes per cell and four stages.  The tiles of two stages that these
// passes replace (k_adj_diff2) spent seven of eight instructions on addresses
// and finished the pole rows in a launch of their own: 512x1024, four stages
// took 58 us, now 20.
#pragma once

#include "sts_march.cuh"

namespace hipft {

struct AdjStage {
  double a, b, c, c0, g, ds;
};

struct AdjPassArgs {
  const double *w0, *w1;  // W_k, W_{k+1}
  const double *y[kMS];   // Y_{k-1}, Y_{k-2}, ...
  double *o0, *o1;        // the last two outputs, the last one in o1
  double *ub, *db;
  AdjStage c[kMS];
  double *dpart;          // [nr][dstride], a slot per warp of the march and per block of the strips
  int dstride;
  int strips, cols;       // theta strips, columns per warp
  const double *dfac;     // [nr+1]
  double bcn, bcs;
  int *err;
};

// Rows at each pole that need its sums within four stages (A^T W takes them in
// rows 1 and 2), rounded to pairs, and the rows a strip owns of the 64 it holds.
// Passes of two stages divide the field in the same way and sum up the D
// partials of each pair of stages by themselves, so that a gradient has the
// same bits however its stages are grouped (stage checkpoints).
constexpr int kJMargin = kMS + 2;
constexpr int kJOwn = 64 - 2 * kJMargin;
constexpr int kJMinRows = 2 * kJMargin;  // smallest ntm of these kernels
constexpr int kJWarps = 2, kJBlocks = 3;  // 64 threads of 255 registers, 69 KB of ring: three blocks per SM
__host__ __device__ constexpr int adj_fields(int ns) { return 4 + ns; }  // W_k, W_{k+1}, ub, db, Y
__host__ __device__ inline size_t adj_march_smem(int ns) {
  return (size_t)kJWarps * (kMSlots * adj_fields(ns) * 64 + kMTab) * sizeof(double);
}
__host__ __device__ inline int adj_strips(int ntm) {
  const int n = (ntm - 2 * kJMargin + kJOwn - 1) / kJOwn;
  return n > 1 ? n : 1;
}
// Columns per warp, as march_cols.
__host__ __device__ inline int adj_cols(int n2, int strips, int nr, int slots) {
  for (int64_t w = 1;; ++w) {
    const int64_t nch = w * slots / ((int64_t)strips * nr);
    if (nch < 1) continue;
    const int64_t c = ((n2 + nch - 1) / nch + kMGroup - 1) / kMGroup * kMGroup;
    if (c <= kMColsMax) return (int)c;
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The rows kJMargin+1 .. ntm-kJMargin, as k_sts_march: at the step that brings
// in column e, stage s works in column e-1-s.  A column's ub and db move on
// with the stages, each of which adds its share; all operands come three
// columns ahead through the ring in shared memory.
template <int NS, typename Off>
__global__ void __launch_bounds__(32 * kJWarps, kJBlocks) k_adj_march(Mesh m, AdjPassArgs a, PairTables pt) {
  extern __shared__ __align__(16) double jsm[];
  constexpr int M = kJMargin, OWN = kJOwn, F = adj_fields(NS);
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npm = m.npm, n2 = npm - 2, ntm = m.ntm, ncol = a.cols;
  const int nch = (n2 + ncol - 1) / ncol, nblk = (nch + kJWarps - 1) / kJWarps;
  const int strip = blockIdx.x % a.strips, rest = blockIdx.x / a.strips;
  const int chunk = (rest % nblk) * kJWarps + warp, i = rest / nblk;  // 0-based
  const int c0 = 2 + chunk * ncol, c1 = min(c0 + ncol - 1, npm - 1);
  if (c0 > npm - 1) {
    pdl_wait();
    return;
  }
  const int r = 1 + OWN * strip + 2 * lane;  // this lane's rows r, r+1
  const double *R = pt.row + (int64_t)i * 3 * pt.LR;  // entry jj holds row jj-1
  auto row = [&](int f, int j) { return R[f * pt.LR + min(j + 1, pt.LR - 1)]; };
  const double2 st = make_double2(row(0, r), row(0, r + 1));
  const double2 c2 = make_double2(row(1, r), row(1, r + 1)), c4 = make_double2(row(2, r), row(2, r + 1));
  const double c2n = row(1, r + 2), c4p = row(2, r - 1);
  const bool own = lane >= M / 2 && lane < 32 - M / 2;
  const bool va = own && r <= ntm - M, vb = own && r + 1 <= ntm - M;

  const int64_t pb = (int64_t)i * m.plane;
  const Off ldb = (Off)m.ldt * 8;
  const Off rowb = (Off)min(r - 1, m.ldt - 2) * 8;
  const char *src[F] = {reinterpret_cast<const char *>(a.w0 + pb), reinterpret_cast<const char *>(a.w1 + pb),
                        reinterpret_cast<const char *>(a.ub + pb), reinterpret_cast<const char *>(a.db + pb)};
#pragma unroll
  for (int s = 0; s < NS; ++s) src[4 + s] = reinterpret_cast<const char *>(a.y[s] + pb);
  const double2 *pt_col = reinterpret_cast<const double2 *>(pt.col) + (int64_t)i * pt.LC;
  char *o0 = reinterpret_cast<char *>(a.o0 + pb), *o1 = reinterpret_cast<char *>(a.o1 + pb);
  char *ub = reinterpret_cast<char *>(a.ub + pb), *db = reinterpret_cast<char *>(a.db + pb);

  constexpr uint32_t kF = 512, kSlot = F * kF;
  double *ring = jsm + (size_t)warp * kMSlots * F * 64, *tab = jsm + (size_t)kJWarps * kMSlots * F * 64 + warp * kMTab;
  const uint32_t sring = smem_addr(ring) + 16u * lane;
  int fc = c0 - NS, left = c1 - c0 + 1 + 2 * NS;
  if (fc < 2) fc += n2;
  Off fo = (Off)(fc - 1) * ldb + rowb;
  auto fetch = [&](uint32_t s) {
    if (left > 0) {
#pragma unroll
      for (int f = 0; f < F; ++f) cp_async16(s + f * kF, src[f] + fo);
    }
    cp_async_commit();
    --left;
    fo += ldb;
    if (++fc > npm - 1) {
      fc = 2;
      fo -= (Off)n2 * ldb;
    }
  };
  for (int t = lane; t < left + kMGroup - 1; t += 32) cp_async16(smem_addr(tab) + 16u * t, pt_col + c0 - NS + t);
  // what the pass before wrote: it has ended, since k_adj_poles, launched directly
  // before this grid, triggers it only behind its own wait for that pass
  fetch(sring);
  fetch(sring + kSlot);
  fetch(sring + 2 * kSlot);

  const bool odd = strip == a.strips - 1 && ((ntm - M) & 1);
  auto put = [&](bool p, char *o, Off off, double2 y) {
    st_if(p && vb, o + off, y);
    if (odd && p && va && !vb) *reinterpret_cast<double *>(o + off) = y.x;
  };
  double2 W[NS][2] = {};
  PhiCoef K[4] = {};
  double2 U[NS] = {}, D[NS] = {};
  double2 Pc = {}, Pm = {};  // table entries of columns e-1, e-2
  double dsx[NS / 2] = {}, dsy[NS / 2] = {};
  int oc = -2 * NS;                               // column e-NS, counted from c0
  Off wo = (Off)(c0 - 1 - 2 * NS) * ldb + rowb;   // its offset
  const int nown = c1 - c0 + 1;
  uint32_t ptab = smem_addr(tab);
  auto step = [&](auto jc, auto nc, uint32_t sa, uint32_t sb) {
    constexpr int j = decltype(jc)::value, n = decltype(nc)::value;  // n: 2 NS and more: all stages
    constexpr int A = j & 1, B = 1 - A;
    auto slot = [&](int back) {
      return j >= back ? sa + (uint32_t)(j - back) * kSlot : sb + (uint32_t)(j - back + kMGroup) * kSlot;
    };
    cp_async_wait<2>();
    fetch(j + 3 < kMGroup ? sa + (j + 3) * kSlot : sb + (j + 3 - kMGroup) * kSlot);
    const double2 x0 = lds2(slot(0));
    if (n == 0) __syncwarp();  // the table was fetched by all lanes
    const double2 P = lds2(ptab);
    ptab += 16;
    if (n >= 2) {
      // c1 of column e, c5 of column e-2, and the diagonal of column e-1
      PhiCoef &q = K[(j + 3) & 3];
      q.c1 = make_double2(P.x * st.x * st.x, P.x * st.y * st.y);
      q.c5 = make_double2(Pm.y * st.x * st.x, Pm.y * st.y * st.y);
      q.c3 = make_double2(-(Pc.x * st.x * st.x + c2.x + c4.x + Pc.y * st.x * st.x),
                          -(Pc.x * st.y * st.y + c2.y + c4.y + Pc.y * st.y * st.y));
    }
    Pm = Pc;
    Pc = P;
    double2 y[NS + 1] = {};
    y[0] = x0;
    double2 un[NS] = {}, dn_[NS] = {};
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      if (n >= 2 * s + 2) {
        const uint32_t sl = slot(s + 1);
        const AdjStage &c = a.c[s];
        const PhiCoef &q = K[(j + 3 - s) & 3];
        const double2 xl = W[s][A], xc = W[s][B], xr = y[s];
        const double up = __shfl_up_sync(0xffffffffu, xc.y, 1), dn = __shfl_down_sync(0xffffffffu, xc.x, 1);
        const double ax = q.c3.x * xc.x + q.c1.x * xr.x + q.c5.x * xl.x + c2.y * xc.y + c4p * up;
        const double ay = q.c3.y * xc.y + q.c1.y * xr.y + q.c5.y * xl.y + c2n * dn + c4.x * xc.x;
        const double2 pv = s ? W[s > 0 ? s - 1 : 0][A] : lds2(sl + kF);
        const double2 yv = lds2(sl + (4 + s) * kF);
        y[s + 1] = make_double2(c.a * xc.x + c.c * ax + c.b * pv.x, c.a * xc.y + c.c * ay + c.b * pv.y);
        const double2 u0 = s ? U[s > 0 ? s - 1 : 0] : lds2(sl + 2 * kF);
        const double2 d0 = s ? D[s > 0 ? s - 1 : 0] : lds2(sl + 3 * kF);
        un[s] = make_double2(u0.x + c.c0 * xc.x, u0.y + c.c0 * xc.y);
        dn_[s] = make_double2(d0.x + c.g * xc.x, d0.y + c.g * xc.y);
        // selected, not multiplied by zero: past the chunk the ring may hold anything, a NaN too
        const int col = oc + NS - 1 - s;
        const bool in = col >= 0 && col < nown;
        dsx[s / 2] += in ? c.ds * (ax * yv.x) : 0.0;
        dsy[s / 2] += in ? c.ds * (ay * yv.y) : 0.0;
      }
    }
    if (n >= 2 * NS - 1) put(oc + 1 < nown, o0, wo + ldb, y[NS - 1]);
    if (n >= 2 * NS) {
      put(oc < nown, o1, wo, y[NS]);
      put(oc < nown, ub, wo, un[NS - 1]);
      put(oc < nown, db, wo, dn_[NS - 1]);
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      W[s][A] = y[s];
      U[s] = un[s];
      D[s] = dn_[s];
    }
    ++oc;
    wo += ldb;
  };
  uint32_t sa = sring, sb = sring + kMGroup * kSlot;
  step(IntC<0>{}, IntC<0>{}, sa, sb);
  step(IntC<1>{}, IntC<1>{}, sa, sb);
  step(IntC<2>{}, IntC<2>{}, sa, sb);
  step(IntC<3>{}, IntC<3>{}, sa, sb);
  if (NS > 2) {
    step(IntC<0>{}, IntC<4>{}, sb, sa);
    step(IntC<1>{}, IntC<5>{}, sb, sa);
    step(IntC<2>{}, IntC<6>{}, sb, sa);
    step(IntC<3>{}, IntC<7>{}, sb, sa);
  } else {
    const uint32_t x = sa;
    sa = sb;
    sb = x;
  }
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
  double *dp = a.dpart + (int64_t)i * a.dstride + strip * nch + chunk;
#pragma unroll
  for (int h = 0; h < NS / 2; ++h) {
    const double ds = warp_sum((va ? dsx[h] : 0.0) + (vb ? dsy[h] : 0.0));
    if (lane == 0) *dp += ds;
  }
  // this grid ends after the strips' grid, so that the next pass has both
  pdl_wait();
}

// The rows 1..kJMargin and ntm-kJMargin+1..ntm, as k_sts_poles: one
// cluster per realization and pole, a column per thread.  Strip row q is theta
// row q+1 or ntm-q; PR rows of the inputs are held and one is lost per stage.
__host__ __device__ inline size_t adj_poles_smem(int ns, int threads) {
  return (size_t)(2 * (kJMargin + ns) + 2 * kJMargin) * poles_stride(threads) * sizeof(double);
}

template <int NS, int NT>
__global__ void __launch_bounds__(NT, 1) k_adj_poles(Mesh m, AdjPassArgs a, PairTables pt) {
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  extern __shared__ __align__(16) double qsm[];
  constexpr int M = kJMargin, PR = M + NS, H = kMS;  // H: halo columns, the same for all NS
  __shared__ double s_sum[NS][8 * (NT / 32)];
  __shared__ double s_row[5][PR];  // st_i, c2, c4, the coefficients of the neighbours towards and off the pole
  __shared__ double s_ds[NS / 2][NT / 32];
  __shared__ uint64_t s_bar[NS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int npm = m.npm, n2 = npm - 2, ntm = m.ntm;
  const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int unit = blockIdx.x / nc, i = unit >> 1;
  const bool south = (unit & 1) != 0;
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&s_bar[s], 1);
      mbar_expect_tx(&s_bar[s], (uint32_t)(nc * nw * 8));
    }
    fence_mbar_init();
  }
  __syncwarp();
  cluster_arrive();  // waited for below: the blocks' barriers are ready
  const int own = (n2 + nc - 1) / nc;
  const int kb = 2 + rank * own, nown = max(0, min(own, npm - kb));
  const int w = nown + 2 * H;
  const int S = poles_stride(blockDim.x);
  double *sX = qsm, *sY = sX + PR * S, *sU = sY + PR * S, *sD = sU + M * S;
  const int64_t ld = m.ldt, pb = (int64_t)i * m.plane;
  auto wrap = [&](int c) {
    while (c < 2) c += n2;
    while (c > npm - 1) c -= n2;
    return c;
  };
  const int c = min(tid, w - 1), cm = max(c - 1, 0), cp = min(c + 1, w - 1);
  const bool mine = tid >= H && tid < H + nown;
  const int k = wrap(kb - H + c);
  const double2 *Pt = reinterpret_cast<const double2 *>(pt.col) + (int64_t)i * pt.LC;
  const double2 P = Pt[k];
  const double c1n = Pt[wrap(k + 1)].x, c5p = Pt[wrap(k - 1)].y;
  const double Dr = a.dfac[i + 1], bc = south ? a.bcs : a.bcn;
  const double Dp = (Dr + Dr) * m.dp[k] * bc;
  if (tid < PR) {
    const int j = south ? ntm - tid : tid + 1;
    const double *R = pt.row + (int64_t)i * 3 * pt.LR;
    s_row[0][tid] = R[j + 1];
    s_row[1][tid] = R[pt.LR + j + 1];
    s_row[2][tid] = R[2 * pt.LR + j + 1];
    const double c2n = j + 1 <= ntm - 1 ? R[pt.LR + j + 2] : 0.0, c4p = j - 1 >= 2 ? R[2 * pt.LR + j] : 0.0;
    s_row[3][tid] = south ? c2n : c4p;
    s_row[4][tid] = south ? c4p : c2n;
  }
  const int64_t g0 = pb + (int64_t)(k - 1) * ld + (south ? ntm - 1 : 0);
  const int dir = south ? -1 : 1;
  pdl_wait();
  pdl_trigger();
  double x[PR], z[PR - 1];
#pragma unroll
  for (int q = 0; q < PR; ++q) x[q] = a.w0[g0 + dir * q];
#pragma unroll
  for (int q = 0; q < PR - 1; ++q) z[q] = a.w1[g0 + dir * q];
  {
    double u[M], d[M];
#pragma unroll
    for (int q = 0; q < M; ++q) {
      u[q] = a.ub[g0 + dir * q];
      d[q] = a.db[g0 + dir * q];
    }
#pragma unroll
    for (int q = 0; q < M; ++q) {
      sU[q * S + tid] = u[q];
      sD[q * S + tid] = d[q];
    }
  }
#pragma unroll
  for (int q = 0; q < PR; ++q) sX[q * S + tid] = x[q];
  __syncthreads();
  cluster_wait();
  double *in = sX, *out = sY;
  double dsum = 0.0;
#pragma unroll 1
  for (int s = 0; s < NS; ++s) {
    const AdjStage sc = a.c[s];
    const double v = warp_sum(mine ? x[0] : 0.0);
    if (lane < nc)
      st_async(cluster_addr(smem_addr(&s_sum[s][rank * nw + warp]), lane), v, cluster_addr(smem_addr(&s_bar[s]), lane));
    double yv[M];
    const double *Yg = a.y[s] + g0;
#pragma unroll
    for (int q = 0; q < M; ++q) yv[q] = Yg[dir * q];
    double ax[PR - 1];
#pragma unroll
    for (int q = 1; q < PR - 1; ++q) {  // rows past PR-2-s are not used any more
      const double st = s_row[0][q];
      const double c3 = -(P.x * st * st + s_row[1][q] + s_row[2][q] + P.y * st * st);
      ax[q] = c3 * x[q] + (c1n * st * st) * in[q * S + cp] + (c5p * st * st) * in[q * S + cm];
      if (q == 1)
        ax[q] = ax[q] + s_row[4][q] * x[q + 1];
      else if (south)
        ax[q] = ax[q] + s_row[3][q] * x[q - 1] + s_row[4][q] * x[q + 1];
      else
        ax[q] = ax[q] + s_row[4][q] * x[q + 1] + s_row[3][q] * x[q - 1];
    }
    ax[0] = s_row[4][0] * x[1];
    if (!mbar_wait_bounded(&s_bar[s], 0, 1u << 22)) atomicExch(a.err, 1);
    double g = 0.0;
    for (int q = lane; q < nc * nw; q += 32) g = g + s_sum[s][q];
    g = warp_sum(g);
    ax[0] = ax[0] - Dp * g;
    ax[1] = ax[1] + Dp * g;
    double y[PR - 1];
#pragma unroll
    for (int q = 0; q < PR - 1; ++q) y[q] = sc.a * x[q] + sc.c * ax[q] + sc.b * z[q];
#pragma unroll
    for (int q = 0; q < M; ++q) {
      sU[q * S + tid] += sc.c0 * x[q];
      sD[q * S + tid] += sc.g * x[q];
      if (mine) dsum += sc.ds * (ax[q] * yv[q]);
    }
#pragma unroll
    for (int q = 1; q < PR - 1; ++q) out[q * S + tid] = y[q];
    if (mine && s >= NS - 2) {
      double *o = (s == NS - 1 ? a.o1 : a.o0) + g0;
#pragma unroll
      for (int q = 0; q < M; ++q) o[dir * q] = y[q];
    }
#pragma unroll
    for (int q = 0; q < PR - 1; ++q) {
      z[q] = x[q];
      x[q] = y[q];
    }
    double *t = in;
    in = out;
    out = t;
    if (s & 1) {  // the D partials of a pair of stages
      dsum = warp_sum(dsum);
      if (lane == 0) s_ds[s / 2][warp] = dsum;
      dsum = 0.0;
    }
    __syncthreads();
  }
  if (mine) {
#pragma unroll
    for (int q = 0; q < M; ++q) {
      a.ub[g0 + dir * q] = sU[q * S + tid];
      a.db[g0 + dir * q] = sD[q * S + tid];
    }
  }
  if (tid == 0) {
    const int nch = (n2 + a.cols - 1) / a.cols;
    double *dp = a.dpart + (int64_t)i * a.dstride + a.strips * nch + (south ? nc : 0) + rank;
    for (int h = 0; h < NS / 2; ++h) {
      double t = 0.0;
      for (int q = 0; q < nw; ++q) t = t + s_ds[h][q];
      *dp += t;
    }
  }
  cluster_arrive_relaxed();  // no block leaves while another may still send to it
  cluster_wait();
}

}  // namespace hipft
